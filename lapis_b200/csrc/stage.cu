// Page-locked staging for the emitted-module ABI (stage.h).
#include "stage.h"

#include <algorithm>
#include <atomic>
#include <condition_variable>
#include <cstring>
#include <exception>
#include <functional>
#include <memory>
#include <mutex>
#include <thread>
#include <type_traits>
#include <vector>

#include <immintrin.h>

namespace lapis_b200 {

namespace {

constexpr size_t PIECE = size_t(512) << 10;   // one copy on the bus: half of this loses 25 % of its rate
constexpr size_t BLOCK = size_t(64) << 10;    // what a host thread takes at a time; the last one of a piece sends it
constexpr int BLOCKS_PER_PIECE = PIECE / BLOCK;
constexpr int SLOTS = 16;                     // 8 MB of page-locked memory per device in use
constexpr int HELPERS = 7;                    // one core copies 12 GB/s out of DRAM, the bus takes 51
constexpr size_t HELPED_BYTES = size_t(256) << 10;  // below: the calling thread alone (waking a helper takes about 10 us)
constexpr size_t DIRECT_BYTES = size_t(1) << 20;    // page-locked arrays of at least this size are copied in place

// Blocks of one transfer, taken in ascending order by whichever thread is free.
struct Job {
  std::function<void(size_t)> block;
  size_t count = 0;
  std::atomic<size_t> next{0}, done{0};
  void work() {
    for (size_t b; (b = next.fetch_add(1)) < count;) {
      block(b);
      done.fetch_add(1, std::memory_order_release);
    }
  }
};

// Threads that sleep until there is a job.  A job is complete whether or not they wake up in time for it, or exist.
// They are detached and the pool is never destroyed: a child process forked after the first large call has no such
// threads to join at its exit.
class HelperPool {
 public:
  void run(const std::shared_ptr<Job> &job, size_t bytes) {
    if (bytes >= HELPED_BYTES) {
      {
        std::lock_guard<std::mutex> lock(m_);
        if (!started_) {
          started_ = true;
          const int n = std::min<int>(HELPERS, (int)std::thread::hardware_concurrency() - 1);
          try {
            for (int i = 0; i < n; ++i) std::thread([this] { loop(); }).detach();
          } catch (const std::exception &) {  // no more threads to be had: those that there are, or the caller alone
          }
        }
        job_ = job;
        ++round_;
      }
      wake_.notify_all();
    }
    job->work();
    while (job->done.load(std::memory_order_acquire) < job->count) std::this_thread::yield();
  }

 private:
  void loop() {
    uint64_t seen = 0;
    for (;;) {
      std::shared_ptr<Job> job;
      {
        std::unique_lock<std::mutex> lock(m_);
        wake_.wait(lock, [&] { return round_ != seen; });
        seen = round_;
        job = job_;
      }
      job->work();
    }
  }
  std::mutex m_;
  std::condition_variable wake_;
  std::shared_ptr<Job> job_;
  uint64_t round_ = 0;
  bool started_ = false;
};

struct Ring {
  std::mutex busy;  // one transfer at a time; a second caller waits
  char *mem = nullptr;
  cudaEvent_t done[SLOTS] = {};
  char *slot(size_t piece) { return mem + (piece % SLOTS) * PIECE; }
  cudaEvent_t event(size_t piece) { return done[piece % SLOTS]; }
};

int ring_of_device(Ring **out, int *device) {
  static Ring rings[64];
  int dev = 0;
  LAPIS_CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) return fail(LAPIS_EBADARG, "device index %d not supported", dev);
  Ring &r = rings[dev];
  std::lock_guard<std::mutex> lock(r.busy);
  if (r.mem == nullptr) {
    LAPIS_CUDA_TRY(cudaHostAlloc(reinterpret_cast<void **>(&r.mem), SLOTS * PIECE, cudaHostAllocPortable));
    for (cudaEvent_t &e : r.done) LAPIS_CUDA_TRY(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
  }
  *out = &r;
  *device = dev;
  return LAPIS_OK;
}

// State of the pieces of one transfer.  Every block of a piece waits until its slot is ready, whether the CUDA calls
// succeed or not, so a failure ends the transfer early instead of leaving a thread behind.
struct Pieces {
  explicit Pieces(size_t n) : count(n), ready(n), left(n), sent(n) {
    for (size_t p = 0; p < n; ++p) {
      ready[p] = 0;
      left[p] = BLOCKS_PER_PIECE;
      sent[p] = 0;
    }
  }
  size_t count;
  std::vector<std::atomic<int>> ready, left, sent;
  std::atomic<int> error{(int)cudaSuccess};
  void note(cudaError_t e) {
    int none = (int)cudaSuccess;
    if (e != cudaSuccess) error.compare_exchange_strong(none, (int)e);
  }
  bool failed() const { return error.load() != (int)cudaSuccess; }
  static void wait(const std::atomic<int> &flag) {
    while (flag.load(std::memory_order_acquire) == 0) std::this_thread::yield();
  }
  int status(const char *what) const {
    const cudaError_t e = (cudaError_t)error.load();
    return e == cudaSuccess ? LAPIS_OK : fail(LAPIS_ECUDA, "%s failed: %s", what, cudaGetErrorString(e));
  }
};

HelperPool &helpers() {
  static HelperPool *pool = new HelperPool;
  return *pool;
}

// The C entry points let no exception out.  Everything that allocates does so before a helper can have seen the job.
template <typename F>
int guarded(const char *what, F &&transfer) {
  try {
    return transfer();
  } catch (const std::exception &e) {
    return fail(LAPIS_ECUDA, "%s failed: %s", what, e.what());
  }
}

// Copies into a slot past the caches: the bus then reads memory instead of another core's dirty lines (a 1.9 MB call:
// 127 -> 103 us).  Slot addresses are 256-byte aligned (parts start on 256 bytes, blocks on 64 KB).
__attribute__((target("avx"))) void copy_streaming(char *to, const char *from, size_t n) {
  size_t i = 0;
  for (; i + 128 <= n; i += 128) {
    const __m256i a = _mm256_loadu_si256(reinterpret_cast<const __m256i *>(from + i));
    const __m256i b = _mm256_loadu_si256(reinterpret_cast<const __m256i *>(from + i + 32));
    const __m256i c = _mm256_loadu_si256(reinterpret_cast<const __m256i *>(from + i + 64));
    const __m256i d = _mm256_loadu_si256(reinterpret_cast<const __m256i *>(from + i + 96));
    _mm256_stream_si256(reinterpret_cast<__m256i *>(to + i), a);
    _mm256_stream_si256(reinterpret_cast<__m256i *>(to + i + 32), b);
    _mm256_stream_si256(reinterpret_cast<__m256i *>(to + i + 64), c);
    _mm256_stream_si256(reinterpret_cast<__m256i *>(to + i + 96), d);
  }
  memcpy(to + i, from + i, n - i);
  _mm_sfence();
}
void copy_to_slot(char *to, const char *from, size_t n) {
  static const bool streaming = __builtin_cpu_supports("avx");
  if (streaming)
    copy_streaming(to, from, n);
  else
    memcpy(to, from, n);
}

bool page_locked(const void *p) {
  cudaPointerAttributes a;
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return a.type == cudaMemoryTypeHost;
}

// A corrupt array may hold offsets whose difference does not fit the type and wraps to a plausible length; between offsets
// that are not negative none does, so a negative offset is looked for beside a negative length.  (Where the offsets of a
// range are negative but ascend, the descent to them lies in a range in front, or pos[0] is not 0.)
template <typename I>
void check_pos(const I *pos, int64_t from, int64_t to, int64_t *max_len, int64_t *bad_row) {
  using U = std::make_unsigned_t<I>;
  I longest = 0, bad = 0;
  for (int64_t i = std::max<int64_t>(from, 1); i < to; ++i) {
    const I len = (I)((U)pos[i] - (U)pos[i - 1]);
    longest = len > longest ? len : longest;
    bad |= len | pos[i];
  }
  if (bad < 0)
    for (int64_t i = std::max<int64_t>(from, 1); i < to; ++i)
      if (pos[i] < pos[i - 1]) {
        *bad_row = i - 1;
        break;
      }
  *max_len = (int64_t)longest;
}

// In range when neither c nor limit - 1 - c has its sign bit set.
template <typename I, typename U>
bool check_crd(const I *crd, int64_t from, int64_t to, int64_t limit) {
  U any = 0;
  const U last = (U)(limit - 1);
  for (int64_t i = from; i < to; ++i) any |= (U)crd[i] | (last - (U)crd[i]);
  return (I)any >= 0;
}

}  // namespace

int Upload::add_part(const void *host, size_t bytes, Check check, int64_t limit) {
  parts_[count_] = Part{static_cast<const char *>(host), bytes, 0, check, limit, bytes >= DIRECT_BYTES && page_locked(host)};
  return count_++;
}

size_t Upload::layout() {
  size_t at = 0;
  for (int pass = 0; pass < 2; ++pass) {  // the staged parts first: their device range is one byte stream
    for (int i = 0; i < count_; ++i)
      if (parts_[i].direct == (pass == 1)) {
        parts_[i].offset = at;
        at += (parts_[i].bytes + 255) & ~(size_t)255;
      }
    if (pass == 0) staged_ = at;
  }
  return at;
}

void Upload::check_range(const Part &p, size_t from, size_t to, Facts *f) {
  int64_t len = 0, bad = -1;
  bool ok = true;
  switch (p.check) {
    case NONE: return;
    case POS32: check_pos(reinterpret_cast<const int32_t *>(p.host), from / 4, to / 4, &len, &bad); break;
    case POS64: check_pos(reinterpret_cast<const int64_t *>(p.host), from / 8, to / 8, &len, &bad); break;
    case CRD32:
      // a limit beyond the type's range leaves only negative indices to refuse
      ok = check_crd<int32_t, uint32_t>(reinterpret_cast<const int32_t *>(p.host), from / 4, to / 4,
                                        std::min<int64_t>(p.limit, (int64_t)1 << 31));
      break;
    case CRD64: ok = check_crd<int64_t, uint64_t>(reinterpret_cast<const int64_t *>(p.host), from / 8, to / 8, p.limit); break;
  }
  f->max_row_len = std::max(f->max_row_len, len);
  if (bad >= 0 && (f->bad_row < 0 || bad < f->bad_row)) f->bad_row = bad;
  f->crd_in_range = f->crd_in_range && ok;
}

int Upload::run(void *device, cudaStream_t st, Facts *facts) {
  return guarded("upload", [&] { return transfer(device, st, facts); });
}

int Upload::transfer(void *device, cudaStream_t st, Facts *facts) {
  Ring *ring = nullptr;
  int dev = 0;
  LAPIS_TRY(ring_of_device(&ring, &dev));
  std::lock_guard<std::mutex> lock(ring->busy);
  char *base = static_cast<char *>(device);
  size_t direct_checked = 0;
  for (int i = 0; i < count_; ++i)
    if (parts_[i].direct) {
      LAPIS_CUDA_TRY(cudaMemcpyAsync(base + parts_[i].offset, parts_[i].host, parts_[i].bytes, cudaMemcpyHostToDevice, st));
      if (parts_[i].check != NONE) direct_checked += parts_[i].bytes;
    }
  Pieces pieces((staged_ + PIECE - 1) / PIECE);
  // blocks: the staged byte stream, then the index arrays that are copied in place and only looked at here
  const size_t staged_blocks = pieces.count * BLOCKS_PER_PIECE;
  size_t blocks = staged_blocks;
  for (int i = 0; i < count_; ++i)
    if (parts_[i].direct && parts_[i].check != NONE) blocks += (parts_[i].bytes + PIECE - 1) / PIECE;
  std::mutex merge;
  auto job = std::make_shared<Job>();
  job->count = blocks;
  job->block = [&](size_t b) {
    Facts f;
    if (b < staged_blocks) {
      const size_t p = b / BLOCKS_PER_PIECE;
      if (b % BLOCKS_PER_PIECE == 0) {
        pieces.note(cudaSetDevice(dev));
        if (p >= SLOTS) Pieces::wait(pieces.sent[p - SLOTS]);
        pieces.note(cudaEventSynchronize(ring->event(p)));  // also the last use in an earlier transfer
        pieces.ready[p].store(1, std::memory_order_release);
      } else {
        Pieces::wait(pieces.ready[p]);
      }
      const size_t from = b * BLOCK, to = std::min(staged_, from + BLOCK), start = p * PIECE;
      for (int i = 0; i < count_ && !pieces.failed(); ++i) {
        const Part &q = parts_[i];
        const size_t lo = std::max(from, q.offset), hi = std::min(to, q.offset + q.bytes);
        if (q.direct || lo >= hi) continue;
        copy_to_slot(ring->slot(p) + (lo - start), q.host + (lo - q.offset), hi - lo);
        check_range(q, lo - q.offset, hi - q.offset, &f);
      }
      if (pieces.left[p].fetch_sub(1, std::memory_order_acq_rel) == 1) {
        if (!pieces.failed()) {
          pieces.note(cudaSetDevice(dev));
          pieces.note(cudaMemcpyAsync(base + start, ring->slot(p), std::min(staged_ - start, PIECE), cudaMemcpyHostToDevice, st));
          pieces.note(cudaEventRecord(ring->event(p), st));
        }
        pieces.sent[p].store(1, std::memory_order_release);
      }
    } else {
      size_t k = b - staged_blocks;
      for (int i = 0; i < count_; ++i) {
        if (!parts_[i].direct || parts_[i].check == NONE) continue;
        const size_t n = (parts_[i].bytes + PIECE - 1) / PIECE;
        if (k < n) {
          check_range(parts_[i], k * PIECE, std::min(parts_[i].bytes, (k + 1) * PIECE), &f);
          break;
        }
        k -= n;
      }
    }
    std::lock_guard<std::mutex> l(merge);
    facts->max_row_len = std::max(facts->max_row_len, f.max_row_len);
    if (f.bad_row >= 0 && (facts->bad_row < 0 || f.bad_row < facts->bad_row)) facts->bad_row = f.bad_row;
    facts->crd_in_range = facts->crd_in_range && f.crd_in_range;
  };
  helpers().run(job, staged_ + direct_checked);
  return pieces.status("upload");
}

static int download(void *host, const void *device, size_t bytes, cudaStream_t st) {
  if (bytes == 0 || (bytes >= DIRECT_BYTES && page_locked(host))) {
    if (bytes > 0) LAPIS_CUDA_TRY(cudaMemcpyAsync(host, device, bytes, cudaMemcpyDeviceToHost, st));
    LAPIS_CUDA_TRY(cudaStreamSynchronize(st));
    return LAPIS_OK;
  }
  Ring *ring = nullptr;
  int dev = 0;
  LAPIS_TRY(ring_of_device(&ring, &dev));
  std::lock_guard<std::mutex> lock(ring->busy);
  Pieces pieces((bytes + PIECE - 1) / PIECE);
  auto request = [&](size_t p) {
    if (p >= pieces.count) return;
    if (!pieces.failed()) {
      const size_t from = p * PIECE;
      pieces.note(cudaMemcpyAsync(ring->slot(p), static_cast<const char *>(device) + from, std::min(bytes - from, PIECE),
                                  cudaMemcpyDeviceToHost, st));
      pieces.note(cudaEventRecord(ring->event(p), st));
    }
    pieces.sent[p].store(1, std::memory_order_release);
  };
  for (size_t p = 0; p < (size_t)SLOTS; ++p) request(p);
  auto job = std::make_shared<Job>();
  job->count = (bytes + BLOCK - 1) / BLOCK;
  for (size_t p = 0; p < pieces.count; ++p) pieces.left[p] = (int)std::min<size_t>(BLOCKS_PER_PIECE, job->count - p * BLOCKS_PER_PIECE);
  job->block = [&](size_t b) {
    const size_t p = b / BLOCKS_PER_PIECE, from = b * BLOCK;
    if (b % BLOCKS_PER_PIECE == 0) {
      pieces.note(cudaSetDevice(dev));
      Pieces::wait(pieces.sent[p]);
      if (!pieces.failed()) pieces.note(cudaEventSynchronize(ring->event(p)));
      pieces.ready[p].store(1, std::memory_order_release);
    } else {
      Pieces::wait(pieces.ready[p]);
    }
    if (!pieces.failed()) memcpy(static_cast<char *>(host) + from, ring->slot(p) + (from - p * PIECE), std::min(bytes - from, BLOCK));
    if (pieces.left[p].fetch_sub(1, std::memory_order_acq_rel) == 1 && p + SLOTS < pieces.count) {
      pieces.note(cudaSetDevice(dev));
      request(p + SLOTS);
    }
  };
  helpers().run(job, bytes);
  return pieces.status("download");
}

int stage_download(void *host, const void *device, size_t bytes, cudaStream_t st) {
  return guarded("download", [&] { return download(host, device, bytes, st); });
}

}  // namespace lapis_b200

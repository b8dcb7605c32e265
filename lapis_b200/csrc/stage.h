// Host <-> device transfers of the emitted-module ABI, whose operands are pageable numpy buffers.
//
// The arrays of a call are laid out one behind the other in one device allocation and travel in pieces through a
// ring of page-locked slots: a piece is copied into a slot (and validated while it is in cache) while the pieces in
// front of it are on the bus.  A few host threads share the pieces; arrays that the caller has page-locked, when
// large, are copied from where they are.
#pragma once
#include "common.h"

namespace lapis_b200 {

class Upload {
 public:
  // What is known of the index arrays after run().
  struct Facts {
    int64_t max_row_len = 0;   // of the pos array
    int64_t bad_row = -1;      // first row whose end precedes its start
    bool crd_in_range = true;  // 0 <= crd[j] < crd_limit for every entry
  };
  int add(const void *host, size_t bytes) { return add_part(host, bytes, NONE, 0); }
  template <typename I>
  int add_pos(const I *host, int64_t count) {
    return add_part(host, (size_t)count * sizeof(I), sizeof(I) == 4 ? POS32 : POS64, 0);
  }
  template <typename I>
  int add_crd(const I *host, int64_t count, int64_t limit) {
    return add_part(host, (size_t)count * sizeof(I), sizeof(I) == 4 ? CRD32 : CRD64, limit);
  }
  // Device bytes needed; fixes the layout.
  size_t layout();
  // Enqueues the copies to `device` (layout() bytes) on `st`.  The host arrays have been read when it returns, except
  // those that are copied in place: these are in use until the stream is synchronised.
  int run(void *device, cudaStream_t st, Facts *facts);
  template <typename T>
  T *at(void *device, int part) const {
    return reinterpret_cast<T *>(static_cast<char *>(device) + parts_[part].offset);
  }

 private:
  enum Check { NONE, POS32, POS64, CRD32, CRD64 };
  struct Part {
    const char *host;
    size_t bytes, offset;
    Check check;
    int64_t limit;
    bool direct;
  };
  static constexpr int MAX_PARTS = 8;
  Part parts_[MAX_PARTS];
  int count_ = 0;
  size_t staged_ = 0;  // device bytes [0, staged_) travel through the slots
  int add_part(const void *host, size_t bytes, Check check, int64_t limit);
  int transfer(void *device, cudaStream_t st, Facts *facts);
  static void check_range(const Part &p, size_t from, size_t to, Facts *f);
};

// Device -> host, current on return (synchronises `st`).
int stage_download(void *host, const void *device, size_t bytes, cudaStream_t st);

}  // namespace lapis_b200

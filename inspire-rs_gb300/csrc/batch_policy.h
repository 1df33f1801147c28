// batch_policy.h -- which form of the one-CTA Respond kernel a batch of at most
// as many queries as SMs takes (capi.cu), kept free of CUDA so that a host-only
// check (tests/native) can exercise it.  Internal; not part of the public header.
#pragma once
#include <cstdint>

namespace ighost {

// The latest device batch of more queries than the cluster kernel takes and at
// most as many as SMs, launched outside a capture; its stream by id (a
// destroyed stream's handle may come back as another stream's).
struct LastBatch {
  bool any = false;
  uint64_t stream = 0;
};

// Queries up to which a batch on `stream` may take the form that has an SM to
// itself: the SM count, or none (0)
//  * while the last such batch, on another stream, still runs (ended() false):
//    batches of this size that overlap do better two CTAs to an SM.  Eight of
//    128 queries take 861 us over two streams so, 949 one after the other with
//    an SM to each query;
//  * when captured into a graph, whose launches may overlap.
// Other work on the GPU is not looked at.  Beside a batch of 2048 queries on
// another stream the form pays all the same (it starts on the SMs that the
// larger batch leaves): with eight of 128 after it 2307 us, 2365 two to an SM.
template <class Ended>
int alone_limit(int sm_count, bool captured, const LastBatch& last, uint64_t stream, Ended&& ended) {
  if (captured) return 0;
  return last.any && last.stream != stream && !ended() ? 0 : sm_count;
}

// Whether a host call's batch of more queries than SMs, whose rows are read and
// responses written over the host link, takes an SM to each query with its whole
// rows staged while they are expanded.  With two CTAs to an SM the rows come in
// four chunks, three of them after the expansion; of few columns the steps that
// follow are too short to cover that, and all of a wave's reads, then all its
// writes, meet on the link.  So / two to an SM, us: 600 queries of 1, 2, 4 columns
// 388 / 445, 392 / 449, 398 / 454; 200 of 4 columns 187 / 185; but 200 of 8
// columns 232 / 212, 1200 of 16 1122 / 1004.
inline bool whole_rows(int gamma, uint32_t n, int sm_count) { return gamma <= 4 && (int64_t)n > sm_count; }

}  // namespace ighost

// serve_policy.h -- the serving loop's two dispatch decisions (serve.cu),
// kept free of CUDA so that a host-only check (tests/native) can exercise
// them.  Internal; not part of the public header.
#pragma once
#include <cstddef>
#include <cstdint>

namespace ighost {

// SMs a batch of n queries is counted for: two per query on the two-CTA cluster
// kernel, one on the one-CTA kernel.  Two of the latter's CTAs share an SM, but
// counting half an SM launches partial batches too early: at 90 % load the
// queue grew (p50 25 ms, 0.26 as it is), at 75 % p99 was 0.37 ms, 0.29 as it is.
inline size_t batch_sms(bool pair, size_t n) { return (pair ? 2 : 1) * n; }

// Batch formation: a full batch goes at once; a partial one goes at once
// while the GPU has idle SMs, else when its oldest query has waited
// `wait_ns` (the batches in flight keep the GPU busy meanwhile).
inline bool launch_batch_now(size_t pending, size_t max_batch, size_t inflight_sm, size_t sm_count,
                             int64_t oldest_waited_ns, int64_t wait_ns) {
  return pending >= max_batch || inflight_sm < sm_count || oldest_waited_ns >= wait_ns;
}

// Kernel choice for a batch of nb queries: the two-CTA cluster kernel (two
// SMs per query, the lower latency) when the batch is at most pair_max
// queries and those SMs are idle, else one CTA per query (the higher rate per
// SM, which a loaded GPU needs: the cluster kernel alone serves 57 % of the
// one-CTA rate, 76 queries in 88 us against 2048 in 1356).  While at most half
// the SMs are busy a cluster batch may exceed the idle SMs by a quarter of the
// SM count (an SM frees about every microsecond).
// Measured, Poisson arrivals at 25 / 50 / 75 / 90 % of 1.53 M queries/s, p50 (p99)
// in ms:
//   this rule            0.118 (0.132)  0.180 (0.27)  0.244 (0.29)  0.258 (0.30)
//   no slack             0.119 (0.134)  0.180 (0.27)  0.245 (0.29)  0.258 (0.31)
//   slack at any load    0.118 (0.133)  0.170 (0.28)  0.243 (0.29)  0.258 (0.30)
//   by batch size alone  0.118 (0.133)  0.142 (0.18)  0.690 (0.90)  0.750 (0.95)
//   one CTA always       0.162 (0.222)  0.196 (0.30)  0.246 (0.29)  0.258 (0.30)
// Either choice made alone loses at one end of the load; the slack itself makes
// no difference beyond what two runs of one rule differ by.
inline bool use_pair_kernel(size_t nb, size_t pair_max, size_t inflight_sm, size_t sm_count) {
  const size_t slack = inflight_sm <= sm_count / 2 ? sm_count / 4 : 0;
  return nb <= pair_max && inflight_sm + 2 * nb <= sm_count + slack;
}

}  // namespace ighost

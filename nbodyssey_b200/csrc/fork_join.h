// Host control flow of a step on two streams; no CUDA, so that every path can
// be run without a device.
#pragma once

namespace nb {

// With `has_side`: `fork` orders the second stream behind the first and `side`
// queues work there.  Then `work` queues the first stream's; it sets its
// argument when it has given the second stream work of its own.  Each part runs
// only when those before it succeeded, but once the second stream may hold work
// of the step, `join` -- which orders the first stream behind it -- runs
// whatever failed: work queued before a failure still writes the step's arrays,
// and whoever waits for the first stream alone must not pass it.  Statuses:
// 0 is success; returns the first other one.
template <typename Fork, typename Side, typename Work, typename Join>
int run_forked(bool has_side, Fork fork, Side side, Work work, Join join) {
  bool used = false;
  int rc = 0;
  if (has_side) {
    rc = fork();
    if (rc == 0) {
      used = true;
      rc = side();
    }
  }
  if (rc == 0) rc = work(&used);
  if (used) {
    const int joined = join();
    if (rc == 0) rc = joined;
  }
  return rc;
}

}  // namespace nb

// What the sims and batches of a process have in flight on each device.
//
// The resident step kernel takes the SMs that it needs for a whole call, and before other kernels: beside three
// more sims, or a batch, the two-kernel steps of all of them overlap instead. us per step of one sim, N sims
// stepping at once, resident / two-kernel (B200):
//   rig 442 x 84 FP64      N = 1 5.4 / 12.3, 2 5.4 / 6.8, 3 5.4 / 4.9, 4 5.4 / 3.7, 8 5.4 / 3.6
//   tank 482 x 242 FP32    N = 1 6.6 / 15.7, 2 6.4 / 8.6, 3 6.4 / 6.0, 4 6.4 / 4.6, 8 6.4 / 4.5
//   tank 742 x 372 FP64    N = 1 9.0 / 19.2, 2 9.2 / 11.0, 3 9.3 / 9.8, 4 9.2 / 9.0, 8 9.2 / 9.0
//   tank 1202 x 602 FP32   N = 1 12.6 / 23.0, 2 12.6 / 14.4, 3 12.6 / 12.5, 4 12.6 / 11.0, 8 12.6 / 11.0
//   2,000 steps of a batch of 24 tunnels (114 ms) beside a stepping tank of 482 x 242: 1,430 ms / 133 ms
#pragma once

#include <cuda_runtime.h>

#include <mutex>
#include <vector>

namespace vl {

// One sim's or batch's work; `end` is recorded behind the work of each call.
struct Work {
  int device = 0;
  cudaEvent_t end = nullptr;
  int weight = 1;         // of kMany
  int calls = 0;          // calls that are still queueing work
  bool queued = false;    // `end` has been recorded and not been seen to have passed
  static constexpr int kMany = 3;
};

class InFlight {
 public:
  static InFlight& of_process();
  void add(Work* w);
  void remove(Work* w);
  // A call of `w` that queues work. The end is recorded before finish().
  void start(Work* w);
  void finish(Work* w);
  // Whether the other sims and batches with work in flight on w's device weigh kMany or more.
  bool many_others(const Work* w);

 private:
  std::mutex m_;
  std::vector<Work*> all_;
};

// A call that queues work, from its construction to the end of the scope.
class InFlightCall {
 public:
  explicit InFlightCall(Work* w) : w_(w) { InFlight::of_process().start(w_); }
  ~InFlightCall() { InFlight::of_process().finish(w_); }
  InFlightCall(const InFlightCall&) = delete;
  InFlightCall& operator=(const InFlightCall&) = delete;

 private:
  Work* w_;
};

}  // namespace vl

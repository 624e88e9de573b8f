// What the caller of a launcher knows about the kernels ahead of the launch in its stream.
#pragma once

namespace gfs_host {

// With programmatic launches a kernel may start once every CTA of its predecessor has called pdl_trigger(). Most kernels
// call pdl_wait() first, so when their successor starts, all that precedes THEM has completed, and only they themselves
// may still be running. Late-waiting kernels (products under `late_wait`, the dQ kernel of the attention backward)
// trigger at their start and wait at their end: when their successor starts, they and the kernel before them may be
// running. That is all, because a late-waiting kernel may only follow one that waited before its trigger. pdl_wait()
// itself always means that everything ahead has completed: a late-waiting kernel does not complete before its predecessor.
//
// The products launched by this thread inside a WithHints scope (the kernels of gemm2.cu and gemm3.cu; the others ignore
// it and wait first):
//   early_b    no kernel that may still be running writes operand B (a weight, which no kernel of a pass
//              writes): its first tiles are fetched ahead of pdl_wait(). For all launches of the scope.
//   late_wait  the preceding kernel has waited before its trigger, writes nothing that this one reads or writes, and reads
//              nothing that this one writes: this one starts on SMs as they become free. For the first programmatic launch
//              of the scope, whatever it is: the promise is about the kernel ahead of the scope, and two late-waiting
//              kernels in a row would leave three running.
// us a pass, without -> with: two blocks of hidden 256, a step as a graph 245 -> 235; twelve of hidden 768, logits of 130
// tokens 580 -> 558, a step of 8 x 1024 tokens 10920 -> 10840, of 4 x 512 with dropout 4562 -> 4536.
struct LaunchHints {
  bool early_b, late_wait;
};
inline LaunchHints& launch_hints() {
  static thread_local LaunchHints h = {false, false};
  return h;
}
struct WithHints {
  LaunchHints before;
  WithHints(bool early_b, bool late_wait) : before(launch_hints()) { launch_hints() = LaunchHints{early_b, late_wait}; }
  ~WithHints() { launch_hints() = LaunchHints{before.early_b, false}; }
  WithHints(const WithHints&) = delete;
  WithHints& operator=(const WithHints&) = delete;
};

}  // namespace gfs_host

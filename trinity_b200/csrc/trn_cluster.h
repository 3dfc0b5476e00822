/*
 * trn_cluster.h — which size a kernel's cluster is launched with, device by
 * device. Host code without CUDA calls (the caller brings them).
 */
#ifndef TRN_CLUSTER_H
#define TRN_CLUSTER_H

#include <atomic>

namespace trn {

constexpr int kClusterMax = 16, kClusterMin = 8;   /* blocks */
constexpr int kClusterDevices = 64;

/* One per kernel. Function attributes and what can be resident belong to a
 * device, so the size found is kept per device; a failure is not kept, nor is
 * a smaller size that stood in for a kept one once. Safe from several threads:
 * they can only find the same size. */
struct ClusterSizes {
  std::atomic<int> size[kClusterDevices] = {};   /* 0: not known */

  /* probe(c): cluster size c allowed on the current device `dev` and able to be
   * resident; launch(c): launched. The largest size for which both hold; false
   * when there is none. */
  template <class Probe, class Launch>
  bool launch(int dev, Probe probe, Launch launch) {
    const bool kept = dev >= 0 && dev < kClusterDevices;
    const int known = kept ? size[dev].load(std::memory_order_relaxed) : 0;
    for (int c = known ? known : kClusterMax; c >= kClusterMin; c >>= 1) {
      if (c != known && !probe(c)) continue;
      if (!launch(c)) continue;
      if (kept && !known) size[dev].store(c, std::memory_order_relaxed);
      return true;
    }
    return false;
  }
};

}  // namespace trn

#endif

// Buffers and barriers of a pipeline of tiles walked by two groups of a CTA's threads.
#pragma once

#ifdef __CUDACC__
#define PTX_RING_HD __host__ __device__
#else
#define PTX_RING_HD
#endif

namespace ptx {

// Where tile i of a CTA goes: the group that takes it, its buffer, and the barrier and the parity of
// the barrier's phase that its copy completes.  One barrier per buffer and group, so that a group
// waits for every phase of its own barriers and for no others.  With one per buffer a group met
// barriers whose previous phase only the other group had waited for; while that one is still open,
// a wait on the next one's parity returns at once, before the tile has come.
struct PipeRing {
  static constexpr int kGroups = 2, kBufs = 3, kBars = kGroups * kBufs;
  static_assert(kBufs % kGroups != 0, "i % kBars names one buffer and one group");
  PTX_RING_HD static constexpr int group(int i) { return i % kGroups; }
  PTX_RING_HD static constexpr int buffer(int i) { return i % kBufs; }
  PTX_RING_HD static constexpr int barrier(int i) { return i % kBars; }
  PTX_RING_HD static constexpr unsigned parity(int i) { return (i / kBars) & 1; }
  // whether tile i's copy has been issued and its group stopped before it: next[g] is the first tile
  // that group g has not finished, and with tile k it issued tile k + kBufs
  PTX_RING_HD static constexpr bool left_open(int i, const int* next) {
    return i >= next[group(i)] && (i < kBufs || i - kBufs < next[group(i - kBufs)]);
  }
};

}  // namespace ptx

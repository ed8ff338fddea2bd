// One value per block of a cluster, brought together in the first block's shared memory.
//
// A block's shared memory may be touched by the others only from the time it is known to have
// started, and co-scheduling does not tell them that: a block that is through with its part first
// could store before the first block runs. So each block arrives at the cluster's barrier when it
// starts and waits there before its store; the work in between hides the barrier. A second barrier
// behind the store says that all values are there, and keeps the first block's memory until then.
#pragma once

#ifdef __CUDACC__
#define XD_MEET_FN __device__ __forceinline__
#else
#define XD_MEET_FN inline
#endif

template <class Cluster>
class ClusterMeet {
 public:
  // At the kernel's start, by all threads of every block. on: the grid is a cluster of several blocks.
  XD_MEET_FN ClusterMeet(Cluster cluster, bool on) : cl(cluster) {
    if (on) cl.barrier_arrive();
  }
  // This block's value (the leader thread's) to slot `rank` of the first block's array. By all
  // threads, once, and only where `on`: the first block may read its slots afterwards.
  template <typename T>
  XD_MEET_FN void put(T v, T *slots, bool leader) {
    cl.barrier_wait();
    if (leader) *cl.map_shared_rank(slots + cl.block_rank(), 0) = v;
    cl.sync();
  }

 private:
  Cluster cl;
};

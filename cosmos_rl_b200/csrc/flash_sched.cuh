// Work list of the attention kernels: (sequence, block of rows, head) items over packed sequences, read from the cumulative
// lengths on the device, the costly ones first.
//
// Order. Under the causal mask a query block costs its index in the sequence, so the list goes by index from the end, then
// by sequence, then by head. Without it a block costs what its sequence is long: the list goes by length in blocks, then
// by sequence, block and head (3600 and 2340 tokens, 16 heads, forward: 162 us, 195 us by index). Blocks that a short
// sequence does not have are not in it. The grid is an upper bound on its length, found from the shapes alone.
//
// The forward and the dQ kernel take items one after the other: the grid has one CTA an item, but a CTA that is near the
// end of its item takes over the next CTA that has not started (cluster launch control) instead of leaving. It keeps its
// TMEM and barriers, and the loads and first products of the next item run under the end of this one. The hardware hands
// items out in order as CTAs ask, so there is no counter to reset and an SM that gets cheap items takes more of them; CTAs
// past the end of the list are taken over and dropped. One warp walks the list and hands items to the other warps through
// a two-slot queue in shared memory.
// Forward, seven sequences of 640 to 1536 tokens, 28 heads: 106 us; 127 us with a CTA that leaves after each item, 118 us
// with one CTA an SM and the list dealt out in advance, forwards and backwards in turn.
#pragma once
#include "sm100.cuh"

namespace b200 {

struct FlashItem {
  int q_beg, len_q, k_beg, len_k;  // the sequence's rows
  int row0, head, valid, b;        // first row of the block inside the sequence; valid = 0 ends the list
};

// Upper bound on the items of B sequences of together at most `total` rows, none longer than `longest`.
inline long long flash_items(int B, long long total, int longest, int rows, int heads) {
  const long long by_longest = (long long)((longest + rows - 1) / rows) * B, by_total = total / rows + B;
  return (by_longest < by_total ? by_longest : by_total) * heads;
}

// All 32 lanes of a warp. `cu` gives the lengths that are cut into blocks of `rows`.
struct FlashList {
  const int* cu;
  int B, rows, heads, levels;
  bool by_length;             // level = blocks of the sequence - 1; otherwise: index of the block
  int level;                  // what is being listed, from levels - 1 down
  int chunk;                  // first sequence of the 32 that `mask` describes
  int last;                   // last block of sequence chunk + lane, -1 without one
  unsigned mask;              // sequences chunk + lane that have a block at this level
  long long base;             // rank of the first item of the chunk

  __device__ __forceinline__ void load() {
    const int b = chunk + (threadIdx.x & 31);
    last = b < B ? min((cu[b + 1] - cu[b] + rows - 1) / rows, levels) - 1 : -1;
  }
  __device__ __forceinline__ void scan() { mask = __ballot_sync(0xffffffffu, by_length ? last == level : last >= level); }
  __device__ __forceinline__ void rewind() {
    level = levels - 1;
    chunk = 0;
    base = 0;
    load();
    scan();
  }
  __device__ __forceinline__ void init(const int* cu_, int B_, int rows_, int heads_, int levels_, bool by_length_) {
    cu = cu_;
    B = B_;
    rows = rows_;
    heads = heads_;
    levels = levels_;
    by_length = by_length_;
    rewind();
  }
  // item `rank` of the list; false past its end. Ranks rise from call to call, or the walk starts again.
  __device__ __forceinline__ bool find(uint32_t rank, int& b, int& block, int& head) {
    if (rank < base) rewind();
    while (level >= 0) {
      const int each = by_length ? (level + 1) * heads : heads;   // items of a sequence here
      const long long here = (long long)__popc(mask) * each;
      if (rank < base + here) {
        const int r = (int)(rank - base), k = r / each, rest = r - k * each;
        block = by_length ? rest / heads : level;
        head = by_length ? rest - block * heads : rest;
        const unsigned lane = threadIdx.x & 31;   // the k-th set bit of the mask
        b = chunk + __ffs(__ballot_sync(0xffffffffu, ((mask >> lane) & 1) && __popc(mask & ((1u << lane) - 1)) == k)) - 1;
        return true;
      }
      base += here;
      chunk += 32;
      if (chunk >= B) {
        chunk = 0;
        if (--level < 0) break;
      }
      if (B > 32) load();
      scan();
    }
    return false;
  }
};

// The items of one CTA, one warp. `slot` is 16 bytes of shared memory for the answers of cluster launch control, announced
// on `bar` (a count of one). Every request is followed by its answer before the CTA leaves, and none follows a refusal.
struct FlashWork {
  FlashList list;
  uint4* slot;
  uint64_t* bar;
  uint32_t rank, answers;
  bool started, pending, refused;

  __device__ __forceinline__ void init(uint4* slot_, uint64_t* bar_) {
    slot = slot_;
    bar = bar_;
    rank = blockIdx.x;
    answers = 0;
    started = pending = refused = false;
  }
  // asks for the next CTA; to be called when the loads of the current item are nearly through
  __device__ __forceinline__ void request() {
    if (pending || refused) return;
    pending = true;
    if ((threadIdx.x & 31) == 0) {
      mbar_arrive_expect_tx(bar, 16);
      clc_try_cancel(slot, bar);
    }
    __syncwarp();
  }
  // false when the answer did not come in time
  __device__ __forceinline__ bool answer() {
    pending = false;
    if (!__all_sync(0xffffffffu, mbar_wait(bar, answers & 1))) return false;
    ++answers;
    refused = !clc_answer(slot, rank);
    fence_proxy_async_smem();   // the slot has been read before the next answer is written there
    __syncwarp();
    return true;
  }
  // 1: sequence, block and head of this CTA's next item; 0: no more; -1: timed out
  __device__ __forceinline__ int next(int& b, int& block, int& head) {
    while (true) {
      if (started) {
        request();
        if (refused) return 0;
        if (!answer()) return -1;
        if (refused) return 0;
      }
      started = true;
      if (list.find(rank, b, block, head)) return 1;
    }
  }
  __device__ __forceinline__ void finish() {
    if (pending) answer();
  }
};

}  // namespace b200

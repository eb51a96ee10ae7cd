// The wait of a long-read strip for the strip above it (pairhmm_long.cuh).  The
// protocol is written against the warp that waits, so that it also compiles for the
// host, where a test drives it with lanes that see the word at different moments.
#pragma once

#ifdef __CUDACC__
#define VD_WARP_FN __device__ __forceinline__
#else
#define VD_WARP_FN inline
#endif

namespace vd {

constexpr long long kLongSpins = 1ll << 25;  // polls of one wait before it gives up (tens of seconds)

// A task's word: boundary blocks published so far (all of them: the task is
// done), which halves left the range, and the buffer its boundary is in.
VD_WARP_FN int task_blocks(unsigned long long v) { return (int)(v & 0x3fffffffull); }
VD_WARP_FN unsigned task_fail(unsigned long long v) { return (unsigned)(v >> 30) & 3u; }
VD_WARP_FN int task_buffer(unsigned long long v) { return (int)(v >> 32); }

// Waits until the warp's word has published `need` blocks and returns it, the same
// value in every lane: what one lane reads goes to all of them.  (The word moves on
// while it is read, so lanes reading it each for themselves may see different counts,
// and what a lane does next -- whether it enters the next wait, which is a collective
// of the warp -- depends on the count.)  After kLongSpins polls, or once another wait
// has given up, the error flag is set and ok is false in every lane.
//
// Warp: load() reads the word with acquire order; stopped() and give_up() read and set
// the error flag; from_leader(v) is one lane's v in every lane, and orders what that
// lane has read before what the others read later.
template <typename Warp>
VD_WARP_FN unsigned long long wait_word(const Warp& w, int need, bool& ok) {
  unsigned long long v = w.from_leader(w.load());
  for (long long spin = 0; task_blocks(v) < need; ++spin) {
    if (spin >= kLongSpins || ((spin & 1023) == 1023 && w.from_leader(w.stopped() ? 1 : 0) != 0)) {
      w.give_up();
      ok = false;
      break;
    }
    w.pause();
    v = w.from_leader(w.load());
  }
  return v;
}

}  // namespace vd

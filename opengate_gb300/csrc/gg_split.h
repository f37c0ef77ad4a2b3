// gg_split.h - rounds and waiting lists of the split kernel's warps (k_spect_split, gg_spect.cu).
// Plain C++ besides the two attributes, so that the bound below is checked on the host over every
// sequence of rounds.
#pragma once

#ifndef __CUDACC__
#define GG_HD
#else
#define GG_HD __host__ __device__
#endif

namespace gg {

// Copies that wait: for their next trial (retry), for an exact trial (open).  Copies
// enter the lists in rounds of first trials only, 32 at most and with fewer than 32
// in either list; the other rounds take copies from the lists and put back no more.
// So both together hold at most 31 + 31 + 32 copies, all of them in `retry` when the
// exact trials of 32 open ones reject them all; `open` itself is emptied from 32 on
// before any other round, so it holds at most 31 + 32.
constexpr int kSplitRetry = 96, kSplitOpen = 64;

enum SplitRound : int { kSplitDone = 0, kSplitExactTrials = 1, kSplitRetries = 2, kSplitFirstTrials = 3 };

// The warp's next round; last: every copy of the batch has begun.  Full rounds as long as
// there is work for them: exact trials before retries before first trials.
GG_HD constexpr SplitRound split_round(int n_retry, int n_open, bool last) {
  if (n_open >= 32 || (last && n_retry == 0)) return n_open == 0 ? kSplitDone : kSplitExactTrials;
  return n_retry >= 32 || last ? kSplitRetries : kSplitFirstTrials;
}

}  // namespace gg

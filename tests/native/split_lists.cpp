// Every sequence of the split kernel's rounds: the most entries that its waiting lists ever hold.
#include <algorithm>
#include <cstdio>
#include <set>
#include <tuple>
#include <vector>

#include "../../opengate_gb300/csrc/gg_split.h"

int main() {
  using State = std::tuple<int, int, bool>;  // retry, open, no copy left to begin
  std::set<State> seen;
  std::vector<State> todo;
  int most_retry = 0, most_open = 0;
  bool ends = false;
  auto go = [&](int nr, int no, bool last) {
    most_retry = std::max(most_retry, nr);
    most_open = std::max(most_open, no);
    if (nr < 256 && no < 256 && seen.insert({nr, no, last}).second) todo.push_back({nr, no, last});
  };
  go(0, 0, false);
  while (!todo.empty()) {
    const auto [nr, no, last] = todo.back();
    todo.pop_back();
    const gg::SplitRound r = gg::split_round(nr, no, last);
    if (r == gg::kSplitDone) {
      if (nr || no || !last) return 2;  // copies left
      ends = true;
    } else if (r == gg::kSplitExactTrials) {
      const int n = std::min(no, 32);
      if (n == 0) return 2;
      for (int a = 0; a <= n; ++a) go(nr + a, no - n, last);
    } else {
      const bool first = r == gg::kSplitFirstTrials;
      if (first && last) return 2;
      const int n = first ? 32 : std::min(nr, 32), left = first ? nr : nr - n;
      if (n == 0) return 2;
      for (int a = 0; a <= n; ++a)  // rejected, left open; the others are settled
        for (int b = 0; a + b <= n; ++b) {
          go(left + a, no + b, last);
          if (first) go(left + a, no + b, true);
        }
    }
  }
  std::printf("%d of %d, %d of %d\n", most_retry, gg::kSplitRetry, most_open, gg::kSplitOpen);
  return ends && most_retry <= gg::kSplitRetry && most_open <= gg::kSplitOpen ? 0 : 1;
}

// A number that a query finds out once: kept when the query succeeds, a guess for this call alone when it does not (the next
// call asks again).  Plain C++.
#pragma once
#include <atomic>

namespace sb200 {

// kept: 0 = not known yet (null: nowhere to keep it); query(int*) -> bool, the number above zero
template <typename Query>
int remember(std::atomic<int>* kept, Query query, int guess) {
  if (kept != nullptr) {
    const int n = kept->load(std::memory_order_relaxed);
    if (n > 0) return n;
  }
  int n = 0;
  if (!query(&n) || n < 1) return guess;
  if (kept != nullptr) kept->store(n, std::memory_order_relaxed);
  return n;
}

}  // namespace sb200

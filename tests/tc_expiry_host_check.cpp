// Host check of the account of matrix products that a block's threads keep (kb::TcPhase), over
// random products that end at once, late or not at all: the threads step through tc_product and
// p2_tc_end as the kernels do, on a model of the mbarrier. Built by tests/test_tc_expiry.py.
#include <cstdio>
#include <random>
#include <vector>

#include "poseidon2_tc.cuh"

int main() {
  std::mt19937_64 g(11);
  constexpr int THREADS = 8, LIMIT = 100;
  long bad = 0, expiries = 0, drained = 0, lost = 0;
  for (int it = 0; it < 20000; it++) {
    std::vector<kb::TcPhase> ph(THREADS);
    int issued = 0;
    double now = 0, ends = 0;  // end of the last product; the ones before have ended
    bool any = false;
    const double late = g() % 3 ? 0.02 : 0.3;
    for (int p = 0; p < 40; p++) {
      bool stop = false;  // __syncthreads_or
      for (const kb::TcPhase& t : ph) stop = stop || t.expired;
      if (stop != any) bad++;
      if (!stop) {
        if (issued && ends > now) bad++;  // a product started beside one that runs
        issued++;
        const double u = double(g() % 1000) / 1000;
        ends = now + (u < late ? (g() % 4 ? double(g() % (3 * LIMIT)) : 1e9) : 1);
        double left = now;
        for (kb::TcPhase& t : ph) {
          if (t.parity != uint32_t(issued - 1 & 1)) bad++;  // everyone waits for this product's phase
          const double from = now + double(g() % 20);
          const bool done = ends <= from + LIMIT;
          t.waited(done);
          any = any || !done;
          left = std::max(left, done ? std::max(from, ends) : from + LIMIT);
        }
        now = left;
      } else {
        now += 5;
      }
    }
    // p2_tc_end: a thread whose wait ran out waits for its phase again
    double freed = now;
    for (const kb::TcPhase& t : ph) {
      if (!t.expired) continue;
      if (t.parity != uint32_t(issued - 1 & 1)) bad++;  // it is the last product's
      freed = std::max(freed, ends <= now + LIMIT ? std::max(now, ends) : now + LIMIT);
    }
    expiries += any;
    if (any && ends <= now + LIMIT) {
      drained++;
      if (freed < ends) bad++;  // freed under a running product
    } else if (any) {
      lost++;
    } else if (ends > now) {
      bad++;
    }
  }
  std::printf("wrong %ld; blocks with an expiry %ld, drained %ld, given up %ld\n", bad, expiries, drained, lost);
  return bad || !drained || !lost;
}

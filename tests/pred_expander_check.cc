// The host side of a packed pred's arrival (graph500_b200/csrc/pred_expander.h)
// without a GPU: the marks and the state of the work come from this program.
// One check per argument; prints "ok" or what was wrong.
#include "pred_expander.h"

#include <stdio.h>
#include <string.h>
#include <sys/resource.h>
#include <time.h>

#include <algorithm>
#include <fstream>
#include <string>

using namespace g500;
using std::chrono::milliseconds;

namespace {

constexpr int64_t N = 1 << 16;
constexpr int CHUNKS = 16;

struct Fixture {
  std::vector<uint32_t> src = std::vector<uint32_t>(N);
  std::vector<int64_t> dst = std::vector<int64_t>(N, 0x5A5A5A5A5A5A5A5A);
  volatile uint32_t ready[CHUNKS] = {};
  Fixture() {
    for (int64_t i = 0; i < N; ++i)
      src[(size_t)i] = i % 7 == 0 ? PACK_NONE : (uint32_t)(i * 2654435761u) % (31u << PACK_BITS);
  }
  void mark(int c, uint32_t run, bool bad = false) {
    std::atomic_thread_fence(std::memory_order_release);
    ready[c] = run << 1 | (bad ? 1u : 0u);
  }
  void mark_all(uint32_t run) {
    for (int c = 0; c < CHUNKS; ++c) mark(c, run);
  }
  bool expanded(int64_t b, int64_t e) const {
    for (int64_t i = b; i < e; ++i) {
      const uint32_t p = src[(size_t)i];
      const int64_t want = p == PACK_NONE ? -1 : (int64_t)(p % (1u << PACK_BITS)) + ((int64_t)(p >> PACK_BITS) << 48);
      if (dst[(size_t)i] != want) return false;
    }
    return true;
  }
};

std::string entries() {
  for (int threads : {1, 3, 16}) {
    Fixture f;
    PredExpander x(threads);
    for (uint32_t run = 1; run <= 20; ++run) {
      std::fill(f.dst.begin(), f.dst.end(), 7);
      std::thread marks([&] {
        for (int c = CHUNKS - 1; c >= 0; --c) f.mark((c + (int)run) % CHUNKS, run);  // in any order
      });
      const bool done = x.run(f.src.data(), f.dst.data(), N, CHUNKS, f.ready, run, [] { return WorkState::running; });
      marks.join();
      if (!done || !f.expanded(0, N)) return "run " + std::to_string(run) + " with " + std::to_string(threads) + " threads";
    }
  }
  return "ok";
}

// work that ends without marking every chunk ends the wait
std::string unmarked() {
  Fixture f;
  PredExpander x(4);
  f.mark(0, 1);
  if (x.run(f.src.data(), f.dst.data(), N, CHUNKS, f.ready, 1, [] { return WorkState::complete; })) return "complete";
  PredExpander y(4, milliseconds(20));
  f.mark(0, 2);
  if (y.run(f.src.data(), f.dst.data(), N, CHUNKS, f.ready, 2, [] { return WorkState::refused; })) return "refused";
  return "ok";
}

// a state refused once near the end of a run that went well says nothing about a later run
std::string refused_once() {
  Fixture f;
  PredExpander x(2, milliseconds(50));
  for (uint32_t run = 1; run <= 2; ++run) {
    int calls = 0;
    // refused at the first query; the marks come with the second
    const bool done = x.run(f.src.data(), f.dst.data(), N, CHUNKS, f.ready, run, [&] {
      if (++calls > 1) f.mark_all(run);
      return calls == 1 ? WorkState::refused : WorkState::complete;
    });
    if (!done) return "run " + std::to_string(run) + " given up after " + std::to_string(calls) + " queries";
    std::this_thread::sleep_for(milliseconds(80));
  }
  return "ok";
}

// a run whose entries do not fit is over for the expander: the caller copies it another way
std::string does_not_fit() {
  for (int threads : {1, 4}) {
    Fixture f;
    PredExpander x(threads);
    for (int c = 0; c < CHUNKS; ++c) f.mark(c, 1, c >= 2);
    if (!x.run(f.src.data(), f.dst.data(), N, CHUNKS, f.ready, 1, [] { return WorkState::running; })) return "given up";
    for (int64_t i = 2 * (N / CHUNKS); i < N; ++i)
      if (f.dst[(size_t)i] != 0x5A5A5A5A5A5A5A5A) return "entry " + std::to_string(i) + " written";
    f.mark_all(2);
    if (!x.run(f.src.data(), f.dst.data(), N, CHUNKS, f.ready, 2, [] { return WorkState::running; }) ||
        !f.expanded(0, N))
      return "the next run";
  }
  return "ok";
}

double cpu_seconds() {
  timespec t;
  clock_gettime(CLOCK_PROCESS_CPUTIME_ID, &t);
  return (double)t.tv_sec + 1e-9 * (double)t.tv_nsec;
}

// while nothing is marked, only the calling thread polls without a break
std::string long_wait() {
  Fixture f;
  PredExpander x(16);
  f.mark_all(1);
  x.run(f.src.data(), f.dst.data(), N, CHUNKS, f.ready, 1, [] { return WorkState::running; });  // every thread is up
  std::thread marks([&] {
    std::this_thread::sleep_for(milliseconds(300));
    f.mark_all(2);
  });
  const double c0 = cpu_seconds();
  const auto t0 = std::chrono::steady_clock::now();
  const bool done = x.run(f.src.data(), f.dst.data(), N, CHUNKS, f.ready, 2, [] { return WorkState::running; });
  const double wall = std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
  const double cpus = (cpu_seconds() - c0) / wall;
  marks.join();
  if (!done || !f.expanded(0, N)) return "entries";
  return cpus < 2.5 ? "ok" : std::to_string(cpus) + " processors busy while nothing had arrived";
}

// where the system gives fewer threads than asked for, those do the work
std::string few_threads() {
  std::ifstream statm("/proc/self/statm");
  long pages = 0;
  statm >> pages;
  // room for two or three more stacks
  const rlimit limit{(rlim_t)pages * 4096 + (24u << 20), RLIM_INFINITY};
  if (setrlimit(RLIMIT_AS, &limit)) return "setrlimit";
  Fixture f;
  PredExpander x(64);
  for (uint32_t run = 1; run <= 3; ++run) {
    std::fill(f.dst.begin(), f.dst.end(), 7);
    f.mark_all(run);
    if (!x.run(f.src.data(), f.dst.data(), N, CHUNKS, f.ready, run, [] { return WorkState::running; }) ||
        !f.expanded(0, N))
      return "run " + std::to_string(run);
  }
  return "ok";
}

}  // namespace

int main(int argc, char** argv) {
  const struct { const char* name; std::string (*check)(); } checks[] = {
      {"entries", entries},
      {"unmarked", unmarked},
      {"refused_once", refused_once},
      {"does_not_fit", does_not_fit},
      {"long_wait", long_wait},
      {"few_threads", few_threads},
  };
  for (const auto& c : checks)
    if (argc > 1 && !strcmp(argv[1], c.name)) {
      const std::string r = c.check();
      puts(r.c_str());
      return r == "ok" ? 0 : 1;
    }
  return 2;
}

// The CTA form's stop word against a runtime whose copies arrive as late as
// they may: no copy reaches the word after it went back to the pool, nor reads
// its source after that was handed out again.
#include <cuda_runtime.h>

#include <cstdio>

#include "pdhg_stop.h"

int main() {
  for (int raised = 0; raised <= 2; ++raised) {
    {
      b2p::StopWord stop;
      stop.create(0);
      if (*stop.get() != 0) return std::puts("not zero"), 1;
      for (int i = 0; i < raised; ++i) stop.raise();
      if (*stop.get() != 0) return std::puts("the copy did not wait"), 1;
    }
    // the page-locked word that the copy reads is the next one's who asks
    for (FakeStream* s : fake().streams)
      if (!s->queue.empty()) return std::puts("work left behind"), 1;
    if (!fake().live.empty()) return std::puts("word not given back"), 1;
    if (fake().faults) return std::puts("copy into freed memory"), 1;
  }
  { b2p::StopWord never; if (never.get()) return std::puts("a word without create()"), 1; }
  std::puts("ok");
  return 0;
}

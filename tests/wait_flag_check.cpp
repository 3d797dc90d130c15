// Host-side check of the words in which expired waits are reported
// (csrc/host/wait_flag.h), over pages of plain memory.  Built and run on the
// CPU by tests/test_wait_flag.py.
#include <cstdio>
#include <cstdlib>
#include <memory>
#include <set>
#include <thread>

#include "../parcomm_b200/csrc/host/wait_flag.h"

static bool g_alive = true;
static int* page() {
  int* p = static_cast<int*>(std::malloc(qf::WaitWords::kPage * sizeof(int)));
  for (size_t i = 0; i < qf::WaitWords::kPage; ++i) p[i] = -1;
  return p;
}
static bool alive(const int*) { return g_alive; }
static int fails(qf::WaitFlag& f) {
  try {
    f.check();
    return 0;
  } catch (const qf::QfError&) {
    return 1;
  }
}

int main() {
  int bad = 0;
  qf::WaitWords words(page, alive);
  {
    qf::WaitFlag a(words), b(words), idle(words);
    bad += fails(a);  // nothing launched
    *a.word() = 1;
    b.word();
    bad += fails(b) + fails(idle);  // another owner's wait
    bad += fails(a) != 1;           // reported once
    bad += fails(a);
    *a.word() = 1;  // left unread
  }
  {
    qf::WaitFlag c(words), d(words);  // the words of a and b, given back
    c.word();
    d.word();
    bad += fails(c) + fails(d);
  }
  {
    std::vector<std::unique_ptr<qf::WaitFlag>> many;
    std::set<int*> seen;
    for (size_t i = 0; i < 3 * qf::WaitWords::kPage + 5; ++i) {
      many.push_back(std::make_unique<qf::WaitFlag>(words));
      seen.insert(many.back()->word());
      bad += fails(*many.back());
    }
    bad += seen.size() != many.size();
  }
  {
    qf::WaitFlag old(words);
    int* before = old.word();
    g_alive = false;  // the page went with its device
    qf::WaitFlag fresh(words);
    int* p = fresh.word();
    g_alive = true;
    bad += p == before || *p != 0;
  }  // old's word belongs to no page now
  std::vector<std::thread> threads;
  std::vector<int> wrong(8, 0);
  for (int t = 0; t < 8; ++t)
    threads.emplace_back([&, t] {
      for (int i = 0; i < 5000; ++i) {
        qf::WaitFlag f(words);
        int* p = f.word();
        wrong[t] += *p != 0;
        if ((i + t) % 3 == 0) {
          *p = 1;
          wrong[t] += fails(f) != 1;
        }
        wrong[t] += fails(f);
      }
    });
  for (auto& t : threads) t.join();
  for (int w : wrong) bad += w;
  std::printf("{\"mismatches\": %d}\n", bad);
  return bad ? 1 : 0;
}

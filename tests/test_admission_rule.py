"""The rule that says which shared searches run before an admission pass (csrc/gst_admission.h),
compiled on the host and run through the server's and the batch driver's loops: whatever
overflows and comes back, every query finishes, and no slot stays free while a query waits."""
import os
import subprocess

import pytest

import build
import gst_b200 as G

SIM = r"""
#include <cstdio>
#include <cstdlib>
#include <deque>
#include "gst_admission.h"
using namespace gst;
struct Q { int kind; int ss; int overflows; };
// args: queries, slots, queries a search covers, server, kinds, seed; every third query (by a
// hash) overflows once or twice
int main(int, char** a) {
  const int n = atoi(a[1]), slots = atoi(a[2]), covers = atoi(a[3]), server = atoi(a[4]), kinds = atoi(a[5]);
  unsigned r = (unsigned)atoi(a[6]) * 2654435761u + 1u;
  auto rnd = [&] { return (r = r * 1664525u + 1013904223u) >> 16; };
  std::deque<Q> pending;
  for (int i = 0; i < n; i++) pending.push_back({(int)(rnd() % kinds), 0, rnd() % 3 ? 0 : 1 + (int)(rnd() % 2)});
  std::deque<Q> active;
  int left = n;
  for (int pass = 0; left > 0; pass++) {
    if (pass > 100 * n) return printf("stuck: %d left, %zu wait\n", left, pending.size()), 1;
    std::vector<Waiting> queue;
    for (const Q& q : pending) queue.push_back({q.kind, q.ss == 1});
    for (int kind : kinds_due(queue, slots - (int)active.size(), server != 0)) {
      int took = 0;
      for (Q& q : pending)
        if (q.ss == 0 && q.kind == kind && took++ < covers) q.ss = 1;
    }
    for (auto it = pending.begin(); it != pending.end() && (int)active.size() < slots;) {
      if (it->ss == 0) {
        if (server) break;
        ++it;
        continue;
      }
      active.push_back(*it);
      it = pending.erase(it);
    }
    if (!pending.empty() && (int)active.size() < slots)
      return printf("%zu of %d slots taken, %zu wait\n", active.size(), slots, pending.size()), 2;
    for (unsigned done = 1 + rnd() % 2; done-- && !active.empty();) {
      Q q = active.front();
      active.pop_front();
      if (q.overflows > 0) {
        q.overflows--;
        q.ss = 0;
        pending.push_front(q);
      } else {
        left--;
      }
    }
  }
  return 0;
}
"""


@pytest.fixture(scope="module")
def sim(tmp_path_factory):
    d = tmp_path_factory.mktemp("sim")
    (d / "sim.cpp").write_text(SIM)
    subprocess.check_call([build.CXX, "-O1", "-std=c++17", "-I", os.path.join(os.path.dirname(G.__file__), "csrc"),
                           str(d / "sim.cpp"), "-o", str(d / "sim")])
    return str(d / "sim")


@pytest.mark.parametrize("server", [1, 0])
@pytest.mark.parametrize("n,slots,covers", [(1, 1, 64), (3, 1, 64), (32, 16, 64), (52, 16, 36), (64, 32, 64), (100, 8, 64),
                                            (150, 5, 21), (40, 64, 64)])
def test_every_query_finishes_and_no_slot_idles(sim, server, n, slots, covers):
    for kinds in (1, 3):
        for seed in range(8):
            r = subprocess.run([sim, *map(str, (n, slots, covers, server, kinds, seed))], capture_output=True, text=True,
                               timeout=60)
            assert r.returncode == 0, (kinds, seed, r.stdout)

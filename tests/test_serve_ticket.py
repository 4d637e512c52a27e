"""The ticket rule of the element-mode request loop (csrc/serve_ticket.h), run
on the host: whatever the ratio of the workers' polls to the dispatcher's, a
ticket that is published is solved, and every worker leaves."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "madmax_b200", "csrc")

MAIN = r"""
#include <cstdio>
#include <cstdlib>
#include <random>
#include <vector>
#include "serve_ticket.h"
using namespace sp;

// W workers and a dispatcher in random turns; the dispatcher polls once in
// `ratio` worker polls, publishes at seeded times and leaves after `limit`
// polls without work
static int run(int W, int ratio, int limit, unsigned seed) {
  std::mt19937 rng(seed);
  long long claim = 0, end = 0;
  bool gone = false;
  int idle = 0, bursts = 6;
  std::vector<ServeWait> wait(W);
  std::vector<char> left(W, 0);
  std::vector<int> solved(10000, 0);
  int alive = W;
  auto claimed = [&] { return claim; };
  auto take = [&] { return claim++; };
  for (long long step = 0; alive; step++) {
    if (step > 200000000) return 4;
    if (!gone && rng() % (unsigned)(W * ratio) == 0) {
      if (bursts && rng() % 4 == 0) {
        end += 7 * (1 + rng() % 5);
        bursts--;
        idle = 0;
      } else if (++idle > limit) {
        gone = true;
      }
    }
    const int i = rng() % W;
    if (left[i]) continue;
    const bool g = gone;
    const long long t = serve_poll(wait[i], g, end, limit, claimed, take);
    if (t >= 0) {
      if (t >= end || solved[t]++) return 1;
      wait[i] = ServeWait();
    } else if (t == SERVE_LOST) {
      return 2;
    } else if (t == SERVE_LEAVE) {
      left[i] = 1;
      alive--;
    }
  }
  // a worker may leave without a ticket before the dispatcher does; with one
  // left all published load cases are solved
  for (long long t = 0; t < end; t++)
    if (solved[t] != 1) return 3;
  return 0;
}

int main() {
  // a ticket taken past the published ones, polled far more often than any
  // dispatcher's limit, then published
  ServeWait w;
  long long claim = 6;
  auto claimed = [&] { return claim; };
  auto take = [&] { return ++claim; };  // another took the last published one
  if (serve_poll(w, false, 7, 100, claimed, take) != SERVE_WAIT || w.ticket != 7) return 10;
  for (int i = 0; i < 8 * 100 * 20; i++)
    if (serve_poll(w, false, 7, 100, claimed, take) != SERVE_WAIT) return 11;
  if (serve_poll(w, false, 14, 100, claimed, take) != 7) return 12;
  // the dispatcher left: so does the worker, and its ticket is free again
  ServeWait v;
  claim = 13;
  if (serve_poll(v, true, 14, 100, claimed, take) != SERVE_LEAVE || v.ticket != 14) return 13;
  // without a ticket it leaves by itself, with one and no dispatcher in the end too
  ServeWait u;
  claim = 20;
  long long n = 0;
  while (serve_poll(u, false, 14, 100, claimed, take) == SERVE_WAIT) n++;
  if (n != 800 || u.ticket != -1) return 14;
  u.ticket = 20;
  u.idle = 0;
  long long r;
  for (n = 0; (r = serve_poll(u, false, 14, 100, claimed, take)) == SERVE_WAIT; n++) {
  }
  if (r != SERVE_LOST || n != 409600) return 15;
  for (int ratio : {1, 4, 16, 40})
    for (unsigned seed = 1; seed <= 40; seed++) {
      // (a limit that the slowest ratio cannot reach between two bursts)
      const int rc = run(2 + seed % 7, ratio, 64, seed);
      if (rc) {
        std::printf("ratio %d seed %u: %d\n", ratio, seed, rc);
        return 20 + rc;
      }
    }
  return 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="no g++")
def test_every_published_ticket_is_solved(tmp_path):
    src, exe = tmp_path / "ticket.cpp", tmp_path / "ticket"
    src.write_text(MAIN)
    subprocess.run(["g++", "-std=c++17", "-O2", "-Wall", "-I", CSRC, str(src), "-o", str(exe)],
                   check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, (r.returncode, r.stdout)

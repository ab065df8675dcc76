"""
How the CTAs of a launch that wait for one another leave it (mmx_leave.h), compiled for the host: whichever of them gave up
a wait and in whichever order they leave, the last one, and only it, is told to write the results, and whether any gave up.
"""
import itertools
import os
import shutil
import subprocess

import pytest

from conftest import ROOT

HARNESS = r'''
#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <thread>
#include <vector>
#include "mmx_leave.h"

// arguments: one text per case, a letter per CTA in the order in which they leave ('g' gave up, '.' did not);
// '@' first: the CTAs leave at once, as threads
int main(int argc, char** argv) {
  for (int k = 1; k < argc; ++k) {
    const char* text = argv[k];
    const bool threads = *text == '@';
    if (threads) ++text;
    std::vector<bool> gave;
    for (; *text; ++text) gave.push_back(*text == 'g');
    std::atomic<unsigned> words[LEAVE_WORDS] = {};
    auto add = [&](int w, unsigned v) { return words[w].fetch_add(v); };
    std::vector<LeaveResult> r(gave.size());
    auto one = [&](size_t i) { r[i] = leave_launch((unsigned)gave.size(), gave[i], add); };
    std::vector<std::thread> pool;
    for (size_t i = 0; i < gave.size(); ++i) {
      if (threads) pool.emplace_back(one, i);
      else one(i);
    }
    for (auto& t : pool) t.join();
    int last = 0, stalled = 0;
    for (const LeaveResult& x : r) {
      last += x.last;
      stalled += x.stalled;
      if (x.stalled && !x.last) return 1;
    }
    std::printf("%d %d\n", last, stalled);
  }
}
'''


@pytest.fixture(scope='module')
def harness(tmp_path_factory):
    if shutil.which('g++') is None:
        pytest.skip('no host compiler')
    d = tmp_path_factory.mktemp('leave')
    src, exe = d / 'leave.cpp', d / 'leave'
    src.write_text(HARNESS)
    subprocess.run(['g++', '-std=c++17', '-pthread', '-I', os.path.join(ROOT, 'macromax_b200', 'csrc'), '-o', str(exe),
                    str(src)], check=True)
    return str(exe)


@pytest.mark.parametrize('at_once', [False, True])
def test_one_writer_that_sees_every_stall(harness, at_once):
    cases = [''.join(c) for n in range(1, 6) for c in itertools.product('g.', repeat=n)]
    if at_once:
        cases = ['@' + c for c in cases * 4]
    out = subprocess.run([harness, *cases], check=True, capture_output=True, text=True).stdout.split('\n')
    for case, line in zip(cases, out):
        assert line == f'1 {int("g" in case)}', case

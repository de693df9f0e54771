"""The host threads that make a result buffer's pages present while the device computes: not for
many small buffers, not holding up a call whose device work is done, not touching contents, and
not failing where the host gives no more threads.  (Compiled here; no GPU.)"""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "sparkx_b200", "csrc")

PROGRAM = r"""
#include "prefault.h"
#include <sys/resource.h>
#include <unistd.h>
#include <chrono>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <string>
using sparx::Prefault;

static char* fresh(size_t bytes) {
  void* p = mmap(nullptr, bytes, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS | MAP_NORESERVE, -1, 0);
  if (p == MAP_FAILED) exit(9);
  madvise(p, bytes, MADV_NOHUGEPAGE);
  return (char*)p;
}
static size_t present(char* p, size_t bytes) {
  std::vector<unsigned char> v(bytes / 4096);
  if (mincore(p, bytes, v.data())) exit(9);
  size_t n = 0;
  for (unsigned char x : v) n += x & 1;
  return n * 4096;
}
int main(int, char** argv) {
  const std::string what = argv[1];
  if (what == "small") {   // 1,000 buffers of 12,000 bytes: 12 MB
    Prefault f;
    std::vector<char*> keep;
    for (int i = 0; i < 1000; ++i) { keep.push_back((char*)malloc(12000)); f.add(keep.back(), 12000); }
    f.start();
    printf("%d\n", (int)f.started());
  } else if (what == "many") {  // 400 buffers of 100,000 bytes: 40 MB
    Prefault f;
    for (int i = 0; i < 400; ++i) f.add(fresh(1 << 20), 100000);
    f.start();
    printf("%d\n", (int)f.started());
  } else if (what == "early") {  // the device is done at once
    const size_t bytes = 1ull << 30;
    char* p = fresh(bytes);
    {
      Prefault f;
      f.add(p, bytes);
      f.start();
    }
    const size_t there = present(p, bytes);
    usleep(300000);  // a thread that had not run yet leaves the pages alone
    printf("%zu %zu\n", there, present(p, bytes));
  } else if (what == "whole") {  // every page, contents as they were
    const size_t bytes = 64ull << 20;
    char* p = fresh(bytes + 8192);
    memset(p + 4096 * 3, 7, 4096);
    {
      Prefault f;
      f.add(p + 100, bytes);
      f.start();
      for (int i = 0; i < 2000 && !f.idle(); ++i) usleep(5000);
    }
    size_t sum = 0;
    const size_t there = present(p + 4096, bytes - 4096);
    for (size_t i = 0; i < bytes; ++i) sum += p[i];
    printf("%zu %zu\n", there, sum);
  } else if (what == "nothreads") {  // no address space for a thread's stack
    char* p = fresh(32ull << 20);
    Prefault f;
    f.add(p, 32ull << 20);
    rlimit r{64ull << 20, 64ull << 20};
    if (setrlimit(RLIMIT_AS, &r)) return 9;
    rlimit st{512ull << 20, 512ull << 20};
    setrlimit(RLIMIT_STACK, &st);
    f.start();
    printf("%d\n", (int)f.started());
  }
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("prefault")
    src, exe = d / "t.cpp", d / "t"
    src.write_text(PROGRAM)
    subprocess.run([shutil.which("g++") or "g++", "-O1", "-std=c++17", "-pthread", "-I", CSRC, "-o", str(exe), str(src)],
                   check=True)

    def run(what):
        r = subprocess.run([str(exe), what], capture_output=True, text=True, timeout=120)
        assert r.returncode == 0, (what, r.returncode, r.stderr)
        return [int(x) for x in r.stdout.split()]
    return run


def test_small_results_start_no_threads(program):
    assert program("small") == [0]


def test_many_buffers_count_by_their_bytes(program):
    assert program("many") == [4]


def test_the_end_does_not_wait_for_the_pages(program):
    there, later = program("early")
    assert there < (1 << 30) // 4 and later == there


def test_all_pages_present_and_contents_kept(program):
    there, total = program("whole")
    assert there == (64 << 20) - 4096 and total == 7 * 4096


def test_a_host_without_threads_goes_on(program):
    (started,) = program("nothreads")
    assert started < 4

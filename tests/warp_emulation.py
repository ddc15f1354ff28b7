"""Runs one warp of a device function on the CPU: 32 host threads as lanes, with
the warp's votes and barriers as thread barriers and nothing else in common, so
that lanes drift apart as far as the function's own barriers let them.

`run(body, main)` compiles device code taken from the library's sources
(`extract`) behind a shim of the CUDA names it uses, and returns what `main`
prints.  It is test infrastructure: it shows what depends on the lanes of a warp
running in step, which a GPU run does not.
"""
import functools
import os
import re
import subprocess
import tempfile

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "lair_gb300", "csrc")

SHIM = r"""
#include <atomic>
#include <barrier>
#include <chrono>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <thread>
#include <vector>
#define __device__
#define __global__
#define __forceinline__ inline
#define __noinline__ __attribute__((noinline))
#define __shared__ static
#define __align__(n) __attribute__((aligned(n)))
struct Index { int x = 0; };
static thread_local Index threadIdx, blockIdx;
static std::barrier<> warp_barrier(32);
static unsigned long long warp_slot[32];
static void lanes_meet() { warp_barrier.arrive_and_wait(); }
template <typename F> static unsigned long long vote(unsigned long long v, F fold) {
  warp_slot[threadIdx.x] = v;
  lanes_meet();
  unsigned long long r = warp_slot[0];
  for (int i = 1; i < 32; ++i) r = fold(r, warp_slot[i]);
  lanes_meet();
  return r;
}
static bool __any_sync(unsigned, bool p) { return vote(p, [](auto a, auto b) { return a | b; }) != 0; }
static bool __all_sync(unsigned, bool p) { return vote(p, [](auto a, auto b) { return a & b; }) != 0; }
template <typename T, typename U> static void atomicCAS(T* p, U old, U v) { T o = (T)old; __atomic_compare_exchange_n(p, &o, (T)v, false, __ATOMIC_SEQ_CST, __ATOMIC_SEQ_CST); }
template <typename T, typename U> static void atomicExch(T* p, U v) { __atomic_store_n(p, (T)v, __ATOMIC_SEQ_CST); }
template <typename F> static void run_warp(F f) {
  std::vector<std::thread> lanes;
  for (int i = 0; i < 32; ++i) lanes.emplace_back([=] { threadIdx.x = i; f(i); });
  for (auto& t : lanes) t.join();
}
"""


def extract(source: str, start: str) -> str:
    """The definition that begins with `start` in a source file, to its closing
    brace in the first column."""
    text = open(os.path.join(CSRC, source)).read()
    at = text.index(start)
    return text[at:re.compile(r"^\};?$", re.M).search(text, at).end()]


@functools.lru_cache(maxsize=None)
def _program(code: str):
    where = tempfile.TemporaryDirectory()
    src, exe = os.path.join(where.name, "warp.cpp"), os.path.join(where.name, "warp")
    with open(src, "w") as f:
        f.write(code)
    cmd = ["g++", "-std=c++20", "-O1", "-ffp-contract=off", "-pthread", "-w", src, "-o", exe]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return where, exe  # the folder lives as long as the program is kept


def run(body: str, main: str, args=()) -> str:
    r = subprocess.run([_program(SHIM + body + main)[1], *map(str, args)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    return r.stdout

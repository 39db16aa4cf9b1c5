"""Kernels whose result may not depend on how a block's threads are scheduled: the kernel's
source, compiled for the host with one thread of the block running at a time up to its next
barrier, in ascending and in descending order."""
import ctypes as C
import os
import re
import subprocess

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), 'covasim_gb300', 'csrc')

HARNESS = r'''
#include <cmath>
#include <condition_variable>
#include <cstdint>
#include <mutex>
#include <thread>
#include <vector>
#define __global__
#define __shared__ static
#define __launch_bounds__(...)
using std::isnan;
struct Dim { unsigned x; };
static thread_local Dim threadIdx;
static Dim blockIdx, gridDim;
static std::mutex mu;
static std::vector<std::condition_variable> cv(1024);
static int turn, stride;   // the thread that runs; +1 or -1
static std::vector<bool> done;
static void pass_on(std::unique_lock<std::mutex>&) {
  const int n = (int)done.size();
  for (int k = 1; k <= n; ++k) {
    const int next = ((turn + k * stride) % n + n) % n;
    if (!done[next]) { turn = next; break; }
  }
  cv[turn].notify_one();
}
static void wait_turn(std::unique_lock<std::mutex>& lk) {
  const int me = (int)threadIdx.x;
  cv[me].wait(lk, [me] { return turn == me; });
}
static void __syncthreads() {
  std::unique_lock<std::mutex> lk(mu);
  pass_on(lk);
  wait_turn(lk);
}
KERNEL
extern "C" void run(int descending, unsigned blocks, const float* rec, const float* dead, const float* inf, int64_t n, double* out) {
  gridDim.x = blocks;
  stride = descending ? -1 : 1;
  for (unsigned b = 0; b < blocks; ++b) {
    blockIdx.x = b;
    done.assign(SUM_THREADS, false);
    turn = descending ? SUM_THREADS - 1 : 0;
    std::vector<std::thread> ts;
    for (int k = 0; k < SUM_THREADS; ++k)
      ts.emplace_back([=] {
        threadIdx.x = (unsigned)k;
        { std::unique_lock<std::mutex> lk(mu); wait_turn(lk); }
        k_outcome_sums(rec, dead, inf, n, out);
        std::unique_lock<std::mutex> lk(mu);
        done[k] = true;
        pass_on(lk);
      });
    for (auto& t : ts) t.join();
  }
}
'''


@pytest.mark.parametrize('descending', [0, 1])
def test_outcome_sums_for_any_order_of_the_threads(tmp_path, descending):
    text = open(os.path.join(CSRC, 'covgpu_copy.cu')).read()
    kernel = re.search(r'constexpr int SUM_THREADS.*?\n}\n', text, flags=re.S).group(0)
    src, lib = tmp_path / 'sums.cpp', tmp_path / 'sums.so'
    src.write_text(HARNESS.replace('KERNEL', kernel))
    subprocess.run(['g++', '-std=c++17', '-O1', '-pthread', '-shared', '-fPIC', '-o', str(lib), str(src)], check=True)
    n, blocks = 700, 2  # every thread of both blocks has an agent
    rng = np.random.default_rng(0)
    inf = rng.integers(1, 100, n).astype(np.float32)
    rec, dead = inf + 9, inf + 20
    out = np.zeros((blocks, 3))
    p = lambda x: x.ctypes.data_as(C.c_void_p)  # noqa: E731
    C.CDLL(str(lib)).run(C.c_int(descending), C.c_uint(blocks), p(rec), p(dead), p(inf), C.c_int64(n), p(out))
    np.testing.assert_array_equal(out.sum(axis=0), [2 * n, float(rec.sum() + dead.sum()), 2 * float(inf.sum())])

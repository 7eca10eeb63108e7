"""k_train (tracer_gb300/csrc/mlp.cu) on host threads: what its threads do when
a bounded wait runs out. The kernel's own source runs, a host thread per CUDA
thread, over stand-ins for the tensor-core and barrier instructions
(tc05.cuh); chosen threads' waits give up at once. Whichever threads those
are, every thread has to come to the kernel's end (none left at a barrier for
one that has gone) and the error word has to be set. No GPU is involved."""
import os
import re
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "tracer_gb300", "csrc")

HOST = r"""
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <algorithm>
#include <chrono>
#include <cmath>
#include <condition_variable>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <thread>
#include <vector>
#include "tracer_gpu.h"
#undef __launch_bounds__
#define __launch_bounds__(...)

static thread_local uint3 threadIdx, blockIdx;
static dim3 blockDim, gridDim;
static std::mutex mtx;
static double wait_limit;
static int fail_first, fail_last, fail_wait;   // threads [first, last) fail their fail_wait-th wait
static thread_local int waits;

struct Bar { int count = 0; unsigned gen = 0; bool all = true, out = true; std::condition_variable cv; };
static Bar bars[16];
static bool meet(int id, int threads, bool mine) {
  std::unique_lock<std::mutex> lk(mtx);
  Bar& b = bars[id];
  b.all = b.all && mine;
  if (++b.count == threads) {
    b.out = b.all;
    b.count = 0;
    b.all = true;
    ++b.gen;
    b.cv.notify_all();
    return b.out;
  }
  const unsigned g = b.gen;
  if (!b.cv.wait_for(lk, std::chrono::seconds(30), [&] { return b.gen != g; })) {
    std::printf("thread %u waits at barrier %d, %d of %d came\n", threadIdx.x, id, b.count, threads);
    std::fflush(stdout);
    std::_Exit(3);
  }
  return b.out;
}
static void __syncthreads() { meet(0, (int)blockDim.x, true); }
static int __syncthreads_and(int p) { return meet(0, (int)blockDim.x, p != 0); }
static void __syncwarp() {}
static float __shfl_xor_sync(unsigned, float v, int) { return v; }
static float __uint_as_float(unsigned u) { float f; std::memcpy(&f, &u, 4); return f; }
static void atomicAdd(float* p, float v) { std::lock_guard<std::mutex> lk(mtx); *p += v; }
static void atomicOr(int* p, int v) { std::lock_guard<std::mutex> lk(mtx); *p |= v; }
using std::max;
using std::min;

struct MBar { unsigned need, left, phase; std::condition_variable cv; };
static std::map<uint64_t*, MBar> mbars;
static void arrive(uint64_t* m) {
  std::lock_guard<std::mutex> lk(mtx);
  MBar& b = mbars[m];
  if (--b.left == 0) { b.left = b.need; ++b.phase; b.cv.notify_all(); }
}

namespace trg {
namespace tc05 {
struct Desc { uint32_t lo, hi; };
constexpr uint32_t kTransA = 1u << 15, kTransB = 1u << 16;
static uint32_t smem_u32(const void*) { return 0; }
static uint32_t core_off(uint32_t row, uint32_t k, uint32_t K) {
  return (row >> 3) * (K >> 3) * 128u + (k >> 3) * 128u + (row & 7u) * 16u + (k & 7u) * 2u;
}
constexpr uint32_t idesc_f16_f32(uint32_t M, uint32_t N) { return (1u << 4) | ((N >> 3) << 17) | ((M >> 4) << 24); }
static Desc desc_of(uint32_t, uint32_t, uint32_t) { return Desc{0, 0}; }
static Desc step(Desc d, uint32_t) { return d; }
static void mma_f16(uint32_t, Desc, Desc, uint32_t, uint32_t) {}
static void commit(uint64_t* m) { arrive(m); }
static void fence_before() {}
static void fence_after() {}
static void fence_proxy_async() {}
static void tmem_alloc(uint32_t* slot, uint32_t) { *slot = 0; }
static void tmem_relinquish() {}
static void tmem_dealloc(uint32_t, uint32_t) {}
static void tmem_ld32(uint32_t, uint32_t (&r)[32]) { std::memset(r, 0, sizeof(r)); }
static void tmem_wait(uint32_t (&)[32]) {}
static void tmem_ld16(uint32_t, float (&v)[16]) { std::memset(v, 0, sizeof(v)); }
static void bar_sync(int id, int threads) { meet(id, threads, true); }
static bool bar_all(int id, int threads, bool mine) { return meet(id, threads, mine); }
static void mbar_init(uint64_t* m, uint32_t count) {
  std::lock_guard<std::mutex> lk(mtx);
  MBar& b = mbars[m];
  b.need = b.left = count;
  b.phase = 0;
}
static void mbar_arrive(uint64_t* m) { arrive(m); }
static bool mbar_wait(uint64_t* m, uint32_t parity) {
  const int t = (int)threadIdx.x;
  if (t >= fail_first && t < fail_last && waits++ == fail_wait) return false;
  std::unique_lock<std::mutex> lk(mtx);
  MBar& b = mbars[m];
  return b.cv.wait_for(lk, std::chrono::duration<double>(wait_limit), [&] { return (b.phase & 1u) != parity; });
}
}  // namespace tc05
namespace mlp {
alignas(1024) uint8_t sm[232448];
}
"""

MAIN = r"""
}  // namespace mlp
}  // namespace trg

template <bool LOSS>
static int run(int rows) {
  using namespace trg::mlp;
  blockDim = dim3(kTrainThreads);
  gridDim = dim3(1);
  std::vector<uint8_t> img(kPackedBytes, 0);
  std::vector<float> in((size_t)rows * kIn, 0.25f), dir((size_t)rows * kOut, 0.5f), w(rows, 1.0f);
  std::vector<float> parts(kWsumParts, 1.0f), part(kPartStride);
  int err = 0;
  std::vector<std::thread> th;
  for (unsigned t = 0; t < (unsigned)kTrainThreads; ++t)
    th.emplace_back([&, t] {
      threadIdx = uint3{t, 0, 0};
      blockIdx = uint3{0, 0, 0};
      k_train<LOSS>(img.data(), in.data(), dir.data(), w.data(), (unsigned)rows, rows, 0ull, 0, parts.data(),
                    (float)rows, part.data(), &err);
    });
  for (auto& t : th) t.join();
  return err;
}
int main(int, char** a) {
  const bool loss = std::atoi(a[1]) != 0;
  fail_first = std::atoi(a[2]);
  fail_last = std::atoi(a[3]);
  fail_wait = std::atoi(a[4]);
  wait_limit = fail_last > fail_first ? 1.0 : 60.0;
  std::printf("err %d\n", loss ? run<true>(600) : run<false>(600));  // five tiles: three of group 0, two of group 1
}
"""


@pytest.fixture(scope="module")
def exe(tmp_path_factory):
    if not os.path.exists("/usr/local/cuda/include/cuda_fp16.h"):
        pytest.skip("no CUDA headers")
    src = open(os.path.join(CSRC, "mlp.cu")).read()
    sizes = re.search(r"namespace mlp \{\n(.*?)\}  // namespace mlp", open(os.path.join(CSRC, "mlp.h")).read(), re.S).group(1)
    body = re.search(r"namespace mlp \{\n(.*?)// Column i of the partials", src, re.S).group(1)
    body = sizes + re.sub(r"// x: n x 7 fp32; out.*?(?=// -+ loss, Adam)", "", body, flags=re.S)  # (not k_forward)
    d = tmp_path_factory.mktemp("waits")
    f, out = d / "waits.cpp", d / "waits"
    f.write_text(HOST + "namespace mlp {\n" + body + MAIN)
    r = subprocess.run(["g++", "-O1", "-std=c++17", "-w", "-pthread", f"-I{CSRC}", f"-I{ROOT}/include",
                        "-I/usr/local/cuda/include", str(f), "-o", str(out)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[:4000]
    return str(out)


# threads [first, last) fail their n-th wait (a tile has ten with the loss, nine without): one thread in either
# group, a warp, half a group, a whole group, the last wait of a tile, the MMA thread; none
@pytest.mark.parametrize("loss,first,last,n,err", [(1, 0, 0, 0, 0), (0, 0, 0, 0, 0), (1, 37, 38, 1, 1),
                                                   (1, 300, 301, 4, 1), (1, 64, 96, 9, 1), (1, 0, 128, 3, 1),
                                                   (1, 256, 512, 12, 1), (0, 37, 38, 1, 1), (1, 512, 513, 5, 1)])
def test_every_thread_reaches_the_end(exe, loss, first, last, n, err):
    r = subprocess.run([exe, str(loss), str(first), str(last), str(n)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    assert r.stdout.strip() == f"err {err}"

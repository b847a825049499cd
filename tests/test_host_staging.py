"""The threads that stage host states (zm_staging.cuh), compiled for the CPU
against a stand-in for the CUDA runtime whose copies happen at once: when the
pinned slots are made and given back, what the threads move, and what is left
after a failure."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

RUNTIME = r"""
#include "zm_staging.cuh"
#include <cassert>
#include <cstdio>
#include <cstdlib>
#include <set>
#include <vector>
using zm::HostStage;
static std::set<void*> pinned;
static std::atomic<int> events{0}, made{0}, copies{0};
static int fail_event = -1, fail_copy = -1;
extern "C" {
cudaError_t cudaHostRegister(void* p, size_t, unsigned) { pinned.insert(p); return cudaSuccess; }
cudaError_t cudaHostUnregister(void* p) { assert(pinned.erase(p) == 1); return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) {
  if (made++ == fail_event) return cudaErrorMemoryAllocation;
  ++events;
  *e = (cudaEvent_t)malloc(1);
  return cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t e) { free(e); --events; return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void*) { *a = {}; return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
  if (copies++ == fail_copy) return cudaErrorUnknown;
  memcpy(d, s, n);
  return cudaSuccess;
}
}
struct Call {  // five fields, the device's copy of each, and the results
  std::vector<std::vector<char>> in, dev, out;
  HostStage::Piece up[5], down[5];
  explicit Call(size_t n) {
    for (int f = 0; f < 5; ++f) {
      const size_t b = f < 4 ? n + f : n / 7 + 1;
      in.emplace_back(b);
      for (size_t q = 0; q < b; ++q) in[f][q] = (char)(q * 31 + f);
      dev.emplace_back(b);
      out.emplace_back(b, (char)99);
    }
    for (int f = 0; f < 5; ++f) {
      up[f] = {in[f].data(), dev[f].data(), in[f].size()};
      down[f] = {out[f].data(), dev[f].data(), in[f].size()};
    }
  }
  bool compute() {
    for (int f = 0; f < 5; ++f)
      for (size_t q = 0; q < dev[f].size(); ++q) {
        if (dev[f][q] != in[f][q]) return false;
        dev[f][q] += 1;
      }
    return true;
  }
  bool right() const {
    for (int f = 0; f < 5; ++f)
      for (size_t q = 0; q < in[f].size(); ++q)
        if (out[f][q] != (char)(in[f][q] + 1)) return false;
    return true;
  }
  bool untouched() const {
    for (auto& f : out)
      for (char c : f)
        if (c != 99) return false;
    return true;
  }
};
#define CHECK(x) do { if (!(x)) { printf("line %d: %s\n", __LINE__, #x); return 1; } } while (0)
"""


def _run(tmp_path, main, extra=""):
    src = tmp_path / "t.cc"
    src.write_text(extra + RUNTIME + "int main() {\n" + main + "\n  return 0;\n}\n")
    exe = tmp_path / "t"
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I/usr/local/cuda/include",
                    "-I" + os.path.join(ROOT, "zhenmode_b200", "csrc"), str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout + r.stderr


def test_slots_are_made_when_they_pay_and_given_back(tmp_path):
    _run(tmp_path, r"""
  {
    HostStage small, middle, large;
    for (int n = 0; n < 100; ++n) CHECK(!small.wanted(1u << 20));
    int first = 0;
    while (!middle.wanted(5u << 20)) ++first;
    CHECK(first == 6);  // the seventh call has moved 35 MB
    CHECK(middle.ready() && middle.wanted(5u << 20) && !middle.wanted(1u << 20));
    CHECK(large.wanted(20u << 20) && large.ready());
    CHECK(pinned.size() == 2 && events > 0);
  }
  CHECK(pinned.empty() && events == 0);
""")


@pytest.mark.parametrize("size", [1, 4095, 512 << 10, (512 << 10) + 1, 3000001])
def test_every_byte_goes_up_and_comes_back(tmp_path, size):
    _run(tmp_path, r"""
  HostStage s;
  CHECK(s.ready());
  for (int n = 0; n < 20; ++n) {
    Call c(%d);
    CHECK(s.run(0, nullptr, c.up, c.down, 5, [&] { return c.compute(); }) == cudaSuccess && c.right());
    Call d(%d);
    CHECK(s.run(0, nullptr, d.up, d.down, 5, [] { return false; }) == cudaSuccess && d.untouched());
  }
""" % (size, size))


@pytest.mark.parametrize("n", [0, 1, 3])
def test_a_failed_event_leaves_nothing_behind(tmp_path, n):
    _run(tmp_path, r"""
  {
    HostStage s;
    fail_event = %d;
    CHECK(!s.ready());
    CHECK(pinned.empty() && events == 0);
    CHECK(s.ready());  // the next call may have them
    Call c(1000000);
    CHECK(s.run(0, nullptr, c.up, c.down, 5, [&] { return c.compute(); }) == cudaSuccess && c.right());
  }
  CHECK(pinned.empty() && events == 0);
""" % n)


def test_no_host_memory_is_no_exception(tmp_path):
    """Nothing of a call needs the heap but its threads; where they cannot be had, the caller does the work alone."""
    _run(tmp_path, r"""
  HostStage s;
  CHECK(s.ready());
  Call c(3000001);
  dry = true;
  const cudaError_t e = s.run(0, nullptr, c.up, c.down, 5, [&] { return c.compute(); });
  dry = false;
  CHECK(e == cudaSuccess && c.right());
""", extra=r"""
#include <cstdlib>
#include <new>
static bool dry = false;
void* operator new(std::size_t n) { if (dry) throw std::bad_alloc(); return std::malloc(n); }
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, std::size_t) noexcept { std::free(p); }
""")


@pytest.mark.parametrize("n", [0, 7, 40])
def test_a_failed_copy_is_returned(tmp_path, n):
    _run(tmp_path, r"""
  HostStage s;
  CHECK(s.ready());
  Call c(3000001);
  fail_copy = %d;
  CHECK(s.run(0, nullptr, c.up, c.down, 5, [&] { return c.compute(); }) == cudaErrorUnknown);
  Call d(3000001);
  fail_copy = -1;
  CHECK(s.run(0, nullptr, d.up, d.down, 5, [&] { return d.compute(); }) == cudaSuccess && d.right());
""" % n)

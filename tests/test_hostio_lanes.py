"""The threaded copies of host arrays (harm_hostio.cu) against a stand-in for the CUDA
runtime whose copies happen only when something waits for them, on the CPU: a copy whose
buffer is taken again too early, or that nobody waits for, shows in the data."""
import os
import shutil
import subprocess

import pytest

from harm_cool_b200 import build as hb

RUNTIME = r"""
#include <cuda_runtime_api.h>
#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <deque>
#include <functional>
#include <mutex>
#include <set>
#include <string>
#include <vector>

namespace harm {
int copy_to_host(int device, cudaStream_t st, void *dst, const void *src, size_t n);
int copy_to_device(int device, cudaStream_t st, void *dst, const void *src, size_t n);
bool utoprim_2d_lanes(const double *U, const double *gcov, const double *gcon, const double *gdet, double *prim,
                      int *ret, long n, double gam, int *rc);
}

struct Stream { int device; long issued = 0, done = 0; std::deque<std::function<void()>> q; };
struct Event { Stream *s = nullptr; long at = 0; };
static std::recursive_mutex mu;
static thread_local int device = 0;
static std::set<char *> pinned_at;
static std::vector<std::pair<char *, size_t>> pinned, on_device[4];
static int direct = 0, made_on[4] = {}, wrong_device = 0;
static std::atomic<int> fail_after{-1};
static void wait(Stream *s, long upto)
{
  std::lock_guard<std::recursive_mutex> g(mu);
  while (s->done < upto && !s->q.empty()) { s->q.front()(); s->q.pop_front(); s->done++; }
}
extern "C" {
void **__cudaRegisterFatBinary(void *) { static void *h; return &h; }
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
cudaError_t cudaGetDevice(int *d) { *d = device; return cudaSuccess; }
cudaError_t cudaSetDevice(int d) { device = d; return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char *cudaGetErrorString(cudaError_t) { return "stand-in"; }
cudaError_t cudaMalloc(void **p, size_t n)
{
  *p = std::calloc(n, 1);
  std::lock_guard<std::recursive_mutex> g(mu);
  on_device[device].push_back({(char *)*p, n});
  made_on[device]++;
  return cudaSuccess;
}
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) { *p = std::calloc(n, 1); return cudaSuccess; }
cudaError_t cudaFree(void *p) { std::free(p); return cudaSuccess; }
cudaError_t cudaFreeHost(void *p) { std::free(p); return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned)
{
  Stream *n = new Stream;
  n->device = device;
  *s = (cudaStream_t)n;
  return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s) { delete (Stream *)s; return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { *e = (cudaEvent_t) new Event; return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t e) { delete (Event *)e; return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s)
{
  std::lock_guard<std::recursive_mutex> g(mu);
  ((Event *)e)->s = (Stream *)s;
  ((Event *)e)->at = ((Stream *)s)->issued;
  return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t e)
{
  if (((Event *)e)->s) wait(((Event *)e)->s, ((Event *)e)->at);
  return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t s) { wait((Stream *)s, ((Stream *)s)->issued); return cudaSuccess; }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes *a, const void *p)
{
  std::memset(a, 0, sizeof *a);
  a->type = cudaMemoryTypeUnregistered;
  for (auto &r : pinned)
    if ((const char *)p >= r.first && (const char *)p < r.first + r.second) a->type = cudaMemoryTypeHost;
  return cudaSuccess;
}
}
static void issue(Stream *s, std::function<void()> f)
{
  std::lock_guard<std::recursive_mutex> g(mu);
  if (s->device != device) wrong_device++;
  s->q.push_back(std::move(f));
  s->issued++;
}
extern "C" cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t st)
{
  if (fail_after >= 0 && fail_after-- == 0) return cudaErrorUnknown;
  for (auto &r : pinned)
    if ((char *)d == r.first || (const char *)s == r.first) direct += n == r.second;
  issue((Stream *)st, [=] { std::memcpy(d, s, n); });
  return cudaSuccess;
}
namespace harm {
int fail_with(int code, const std::string &) { return code; }
// the "inversion": prim = 2 U + guess, ret = the zone's first U
void launch_utoprim_batch(cudaStream_t st, const double *U, const double *, const double *, const double *, double *prim,
                          int *ret, long n, double)
{
  issue((Stream *)st, [=] {
    for (long z = 0; z < n; z++) {
      for (int k = 0; k < 8; k++) prim[8 * z + k] += 2 * U[8 * z + k];
      ret[z] = (int)U[8 * z];
    }
  });
}
}  // namespace harm
using namespace harm;
static int bad = 0;
#define EXPECT(c) do { if (!(c)) { std::printf("line %d: %s\n", __LINE__, #c); bad = 1; } } while (0)

static const size_t N = 37u << 20;
static std::vector<char> pattern(size_t n, int seed)
{
  std::vector<char> v(n);
  for (size_t k = 0; k < n; k++) v[k] = (char)((k * 2654435761u >> 7) + seed);
  return v;
}
struct Batch {
  long n;
  std::vector<double> U, gcov, gcon, gdet, prim;
  std::vector<int> ret;
  explicit Batch(long m, int seed) : n(m), U(8 * m), gcov(16 * m), gcon(16 * m), gdet(m), prim(8 * m, 0.5), ret(m, -1)
  {
    for (long z = 0; z < n; z++)
      for (int k = 0; k < 8; k++) U[8 * z + k] = (double)((z + seed) % 100003) + 0.125 * k;
  }
  bool call(int *rc) { return utoprim_2d_lanes(U.data(), gcov.data(), gcon.data(), gdet.data(), prim.data(), ret.data(), n, 1., rc); }
  bool right() const
  {
    for (long z = 0; z < n; z++) {
      if (ret[z] != (int)U[8 * z]) return false;
      for (int k = 0; k < 8; k++)
        if (prim[8 * z + k] != 0.5 + 2 * U[8 * z + k]) return false;
    }
    return true;
  }
};

int main(int argc, char **argv)
{
  const std::string what = argv[1];
  cudaStream_t st;
  cudaStreamCreateWithFlags(&st, 0);
  std::vector<char> dev(N), host = pattern(N, 1), back(N);
  if (what == "copies") {
    for (size_t n : {(size_t)1000, (size_t)(10u << 20) - 8, (size_t)(10u << 20), (size_t)(12u << 20) + 8,
                     (size_t)(20u << 20) - 8, (size_t)(20u << 20), N}) {
      std::fill(dev.begin(), dev.end(), 0);
      EXPECT(copy_to_device(0, st, dev.data(), host.data(), n) == 0);
      cudaStreamSynchronize(st);
      EXPECT(!std::memcmp(dev.data(), host.data(), n));
      std::fill(back.begin(), back.end(), 0);
      EXPECT(copy_to_host(0, st, back.data(), dev.data(), n) == 0);
      EXPECT(!std::memcmp(back.data(), host.data(), n));
    }
    for (long n : {1L, 2048L, 2049L, 5000L, 33000L, 170001L}) {
      Batch b(n, 3);
      int rc = -1;
      EXPECT(b.call(&rc) && rc == 0 && b.right());
    }
  } else if (what == "pinned") {
    pinned.push_back({host.data(), N});
    pinned.push_back({back.data(), N});
    EXPECT(copy_to_device(0, st, dev.data(), host.data(), N) == 0);
    cudaStreamSynchronize(st);
    EXPECT(copy_to_host(0, st, back.data(), dev.data(), N) == 0);
    EXPECT(back == host);
    EXPECT(direct == 2);
    EXPECT(made_on[0] == 0);
  } else if (what == "device") {
    // lanes of device 1 from a thread whose device is 0
    device = 1;
    cudaStream_t st1;
    cudaStreamCreateWithFlags(&st1, 0);
    device = 0;
    EXPECT(copy_to_device(1, st1, dev.data(), host.data(), N) == 0);
    EXPECT(device == 0 && made_on[0] == 0 && made_on[1] > 0);
    EXPECT(copy_to_host(1, st1, back.data(), dev.data(), N) == 0);
    EXPECT(back == host && device == 0 && wrong_device == 0);
  } else if (what == "errors") {
    // whichever copy fails, the next call is whole
    for (int k = 0; k < 24; k++) {
      fail_after = k;
      const int rc = copy_to_device(0, st, dev.data(), host.data(), N);
      const bool hit = fail_after < 0;
      fail_after = -1;
      EXPECT((rc != 0) == hit);
      host = pattern(N, 7 * k);
      EXPECT(copy_to_host(0, st, back.data(), host.data(), N) == 0);
      EXPECT(back == host);
      fail_after = k;
      copy_to_host(0, st, back.data(), dev.data(), N);
      fail_after = -1;
      Batch b(170001, k);
      int rb = -1;
      EXPECT(b.call(&rb) && rb == 0 && b.right());
      fail_after = k;
      Batch f(170001, 2 * k);
      EXPECT(f.call(&rb));
      EXPECT((rb != 0) == (fail_after < 0));
      fail_after = -1;
      Batch one(2000, k);
      EXPECT(one.call(&rb) && rb == 0 && one.right());
      fail_after = k;
      Batch only(2000, k);
      only.call(&rb);
      fail_after = -1;
      std::fill(dev.begin(), dev.end(), 0);
      EXPECT(copy_to_device(0, st, dev.data(), host.data(), N) == 0);
      EXPECT(dev == host);
    }
  }
  std::puts(bad ? "BAD" : "OK");
  std::fflush(stdout);
  std::_Exit(bad);
}
"""


@pytest.fixture(scope="module")
def driver(tmp_path_factory):
    if not os.path.exists(hb.NVCC) and not shutil.which(hb.NVCC):
        pytest.skip("no nvcc")
    d = tmp_path_factory.mktemp("lanes")
    inc = ["-I" + os.path.join(hb.ROOT, "include"), "-I" + hb.CSRC]
    hb._run([hb.NVCC] + hb.ARCH + ["-O2", "-std=c++17", "-w", "-c", os.path.join(hb.CSRC, "harm_hostio.cu"), "-o",
                                   str(d / "hostio.o")] + inc)
    (d / "runtime.cpp").write_text(RUNTIME)
    cuda = os.path.join(os.path.dirname(os.path.dirname(shutil.which(hb.NVCC) or hb.NVCC)), "include")
    hb._run(["g++", "-O2", "-std=c++17", "-I" + cuda, str(d / "runtime.cpp"), str(d / "hostio.o"), "-o",
             str(d / "lanes"), "-lpthread"])
    return str(d / "lanes")


@pytest.mark.parametrize("what", ["copies", "pinned", "device", "errors"])
def test_lanes(what, driver):
    r = subprocess.run([driver, what], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr

// A host's arrays are pageable, and the driver copies pageable memory on one
// thread through a buffer of its own: 4.3 GB/s to a fresh array (its pages are
// faulted in on the way), 9 GB/s from one, of the link's 55 GB/s.  Here up to
// HOST_LANES threads each move every HOST_LANES-th chunk through two pinned buffers
// of their own, so that page faults, host copies and the link overlap.  On 16 host
// cores: reading back 288x256x256 (1.25 GB) 290 -> about 55 ms, Utoprim_2d of
// 100,003 host zones (46 MB) 10.5 -> 2.5 ms.  An array the caller has pinned goes in one
// copy (1.25 GB 23 ms; through the lanes 32).
//
// The lanes of a device are made by the first large copy there (64 MB pinned and
// as much on the device at most, held until the process ends) and belong to one
// call at a time; a call that finds them taken, or a machine that has no room for
// them, copies plainly.
#include "harm_hostio.cuh"

#include <algorithm>
#include <cstring>
#include <exception>
#include <mutex>
#include <thread>

namespace harm {

namespace {
constexpr int MAX_DEVICES = 16;
// Below these the threads cost more than they save (ms, plain against lanes): to the
// device 8.5 MB 0.47, 0.49, 9.7 MB 0.53, 0.50, 16.6 MB 0.86, 0.68; to the host, where now
// and then a thread wakes late, 8.5 MB 0.47, 0.57 to 0.78, 16.6 MB 0.86, 0.69 to 1.02,
// 21 MB 1.08, 0.79 to 0.97.
constexpr size_t TO_DEVICE_MIN = 10u << 20, TO_HOST_MIN = 20u << 20;

struct Slot {
  std::mutex held;
  HostLanes lanes;
  bool made = false, failed = false;
};

Slot &slot(int device)
{
  static Slot *s = new Slot[MAX_DEVICES];  // outlives every caller; the process's end takes it
  return s[device];
}
// memory the driver knows (pinned, managed) goes over the link as it is, in one copy
bool pageable(const void *p)
{
  cudaPointerAttributes a;
  if (cudaPointerGetAttributes(&a, p) == cudaSuccess) return a.type == cudaMemoryTypeUnregistered;
  cudaGetLastError();
  return true;
}
}  // namespace

bool HostLanes::init(int device)
{
  device_ = device;
  n_ = 0;
  OnDevice on(device);
  const int want = std::max(1, std::min<int>(HOST_LANES, (int)std::thread::hardware_concurrency()));
  for (int k = 0; k < want; k++) {
    HostLane &l = lane[k];
    std::memset(&l, 0, sizeof l);
    bool ok = cudaStreamCreateWithFlags(&l.st, cudaStreamNonBlocking) == cudaSuccess;
    for (int b = 0; b < 2 && ok; b++)
      ok = cudaEventCreateWithFlags(&l.done[b], cudaEventDisableTiming) == cudaSuccess &&
           cudaMallocHost(&l.pin[b], LANE_BYTES) == cudaSuccess && cudaMalloc(&l.dev[b], LANE_BYTES) == cudaSuccess;
    if (!ok) {
      for (int b = 0; b < 2; b++) {
        if (l.done[b]) cudaEventDestroy(l.done[b]);
        if (l.pin[b]) cudaFreeHost(l.pin[b]);
        if (l.dev[b]) cudaFree(l.dev[b]);
      }
      if (l.st) cudaStreamDestroy(l.st);
      cudaGetLastError();
      break;
    }
    n_++;
  }
  return n_ > 0;
}

HostLanes *HostLanes::hold(int device)
{
  if (device < 0 || device >= MAX_DEVICES) return nullptr;
  Slot &s = slot(device);
  if (!s.held.try_lock()) return nullptr;
  if (!s.made && !s.failed) {
    s.made = s.lanes.init(device);
    s.failed = !s.made;
  }
  if (!s.made) {
    s.held.unlock();
    return nullptr;
  }
  return &s.lanes;
}

void HostLanes::release() { slot(device_).held.unlock(); }

template <class Body>
cudaError_t HostLanes::run(const Body &body, long parts)
{
  const int n = (int)std::min<long>(n_, parts);
  cudaError_t err[HOST_LANES];
  OnDevice on(device_);  // and the caller's again
  auto one = [&](int k) {
    err[k] = cudaSetDevice(device_);
    if (err[k] == cudaSuccess) err[k] = body(lane[k], k);
  };
  std::thread t[HOST_LANES];
  int started = 1;
  try {
    for (; started < n; started++) t[started] = std::thread(one, started);
  } catch (const std::exception &) {
    // no more threads, or memory for them: the caller takes the remaining lanes' parts too
  }
  one(0);
  for (int k = started; k < n; k++) one(k);
  for (int k = 1; k < started; k++) t[k].join();
  const cudaError_t *bad = std::find_if(err, err + n, [](cudaError_t e) { return e != cudaSuccess; });
  if (bad == err + n) return cudaSuccess;
  // a lane that stopped early left work in flight on its buffers: not into the next call
  for (int k = 0; k < n; k++) cudaStreamSynchronize(lane[k].st);
  return *bad;
}

#define LANE(call)                                \
  do {                                            \
    const cudaError_t e_ = (call);                \
    if (e_ != cudaSuccess) return e_;             \
  } while (0)

int copy_to_host(int device, cudaStream_t st, void *dst, const void *src, size_t n)
{
  if (n >= TO_HOST_MIN && pageable(dst)) {
    HoldLanes h(device);
    if (h.L) {
      CK(cudaStreamSynchronize(st));  // the layout kernel before; the lanes' streams need no event then
      const size_t per = LANE_BYTES, nc = (n + per - 1) / per;
      const int nl = h.L->n();
      CK(h.L->run([&](HostLane &l, int k) {
        size_t before = nc;  // the chunk in flight behind the one being issued
        int b = 0;
        for (size_t c = k; c < nc + nl; c += nl) {
          if (c < nc) {
            LANE(cudaMemcpyAsync(l.pin[b], (const char *)src + c * per, std::min(per, n - c * per),
                                 cudaMemcpyDeviceToHost, l.st));
            LANE(cudaEventRecord(l.done[b], l.st));
          }
          if (before < nc) {
            LANE(cudaEventSynchronize(l.done[b ^ 1]));
            std::memcpy((char *)dst + before * per, l.pin[b ^ 1], std::min(per, n - before * per));
          }
          before = c;
          b ^= 1;
        }
        return cudaSuccess;
      }, (long)nc));
      return HARM_OK;
    }
  }
  CK(cudaMemcpyAsync(dst, src, n, cudaMemcpyDeviceToHost, st));
  CK(cudaStreamSynchronize(st));
  return HARM_OK;
}

int copy_to_device(int device, cudaStream_t st, void *dst, const void *src, size_t n)
{
  if (n >= TO_DEVICE_MIN && pageable(src)) {
    HoldLanes h(device);
    if (h.L) {
      CK(cudaStreamSynchronize(st));  // earlier readers of dst
      const size_t per = LANE_BYTES, nc = (n + per - 1) / per;
      const int nl = h.L->n();
      CK(h.L->run([&](HostLane &l, int k) {
        int b = 0;
        for (size_t c = k; c < nc; c += nl, b ^= 1) {
          const size_t m = std::min(per, n - c * per);
          LANE(cudaEventSynchronize(l.done[b]));
          std::memcpy(l.pin[b], (const char *)src + c * per, m);
          LANE(cudaMemcpyAsync((char *)dst + c * per, l.pin[b], m, cudaMemcpyHostToDevice, l.st));
          LANE(cudaEventRecord(l.done[b], l.st));
        }
        return cudaStreamSynchronize(l.st);
      }, (long)nc));
      return HARM_OK;
    }
  }
  CK(cudaMemcpyAsync(dst, src, n, cudaMemcpyHostToDevice, st));
  return HARM_OK;
}

// Chunks of zones, each packed into a lane's pinned buffer (U, gcov, gcon, gdet,
// prim, and room for ret), inverted on the lane's device buffer and unpacked while
// the next is on its way: one copy each way and no allocation per call.
bool utoprim_2d_lanes(const double *U, const double *gcov, const double *gcon, const double *gdet, double *prim,
                      int *ret, long n, double gam, int *rc)
{
  int device = 0;
  if (cudaGetDevice(&device) != cudaSuccess) return false;
  HoldLanes h(device);
  if (!h.L) return false;
  constexpr long ZONE = 50 * sizeof(double);  // 49 doubles and ret
  constexpr long MOST = (long)(LANE_BYTES / ZONE) / 128 * 128;
  // two chunks a lane where the batch is large enough, to overlap copies with packing
  const int nl = h.L->n();
  const long per = std::min(MOST, std::max(2048L, (n / (2 * nl) + 127) / 128 * 128));
  const long nc = (n + per - 1) / per;
  const cudaError_t e = [&] {
    auto body = [&](HostLane &l, int k) -> cudaError_t {
      long before = nc;
      int b = 0;
      for (long c = k; c < nc + nl; c += nl) {
        if (c < nc) {
          const long z = c * per, m = std::min(per, n - z);
          double *P = (double *)l.pin[b], *D = (double *)l.dev[b];
          std::memcpy(P, U + z * 8, m * 64);
          std::memcpy(P + 8 * m, gcov + z * 16, m * 128);
          std::memcpy(P + 24 * m, gcon + z * 16, m * 128);
          std::memcpy(P + 40 * m, gdet + z, m * 8);
          std::memcpy(P + 41 * m, prim + z * 8, m * 64);
          LANE(cudaMemcpyAsync(D, P, 49 * m * 8, cudaMemcpyHostToDevice, l.st));
          launch_utoprim_batch(l.st, D, D + 8 * m, D + 24 * m, D + 40 * m, D + 41 * m, (int *)(D + 49 * m), m, gam);
          LANE(cudaGetLastError());
          LANE(cudaMemcpyAsync(P + 41 * m, D + 41 * m, m * 68, cudaMemcpyDeviceToHost, l.st));
          LANE(cudaEventRecord(l.done[b], l.st));
        }
        if (before < nc) {
          const long z = before * per, m = std::min(per, n - z);
          const double *P = (const double *)l.pin[b ^ 1];
          LANE(cudaEventSynchronize(l.done[b ^ 1]));
          std::memcpy(prim + z * 8, P + 41 * m, m * 64);
          std::memcpy(ret + z, P + 49 * m, m * 4);
        }
        before = c;
        b ^= 1;
      }
      return cudaSuccess;
    };
    return h.L->run(body, nc);
  }();
  *rc = e == cudaSuccess ? HARM_OK
                         : fail_with(HARM_E_CUDA, std::string("harm_utoprim_2d_batch: ") + cudaGetErrorString(e));
  return true;
}

}  // namespace harm

// Copies between a host's pageable arrays and the device, by several threads
// through pinned buffers (harm_hostio.cu).
#pragma once
#include "harm_common.cuh"

namespace harm {

constexpr int HOST_LANES = 8;              // threads that share a copy
constexpr size_t LANE_BYTES = 4u << 20;    // a lane's buffer (two of them, pinned, and two on the device)

// One thread's part: a stream and two buffers; done[b] is recorded behind the
// device work that last used buffer b.
struct HostLane {
  cudaStream_t st;
  cudaEvent_t done[2];
  char *pin[2], *dev[2];
};

// The lanes of one device, held by one call at a time.  hold() gives null where
// another call holds them or they cannot be had: the caller then copies plainly.
class HostLanes {
public:
  static HostLanes *hold(int device);
  void release();
  int n() const { return n_; }
  // body(lane, index) on every lane, or on as many as there are parts to a call, each
  // on a thread of its own (the first on the caller's) with the device current; the first
  // error, with nothing left in flight after one
  template <class Body>
  cudaError_t run(const Body &body, long parts);

  HostLane lane[HOST_LANES];

private:
  bool init(int device);
  int n_ = 0, device_ = 0;
};

struct HoldLanes {
  HostLanes *L;
  explicit HoldLanes(int device) : L(HostLanes::hold(device)) {}
  ~HoldLanes()
  {
    if (L) L->release();
  }
};

// n bytes from the device to the host after the work on st; dst is complete on return
int copy_to_host(int device, cudaStream_t st, void *dst, const void *src, size_t n);
// n bytes from the host to the device, for later work on st; src is free on return
int copy_to_device(int device, cudaStream_t st, void *dst, const void *src, size_t n);
// Utoprim_2d over n host zones through the lanes; false where they cannot be held
bool utoprim_2d_lanes(const double *U, const double *gcov, const double *gcon, const double *gdet, double *prim,
                      int *ret, long n, double gam, int *rc);
// the batch kernel on device arrays (harm_api.cu)
void launch_utoprim_batch(cudaStream_t st, const double *U, const double *gcov, const double *gcon, const double *gdet,
                          double *prim, int *ret, long n, double gam);

}  // namespace harm

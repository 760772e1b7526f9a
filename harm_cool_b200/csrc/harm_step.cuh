// Kernels of one step that differ between the FP64 path and the mixed path:
// the face fluxes, the update with flux-CT, and the flux diagnostics.
// Included by harm_exact.cu (HARM_STEP_MIXED 0) and harm_mixed.cu (HARM_STEP_MIXED 1),
// each inside its own namespace.
//
// FP64 path: everything in double, built with -fmad=false, bit-compatible
// with the reference.  Mixed path: slopes, face states, the face metric,
// get_state/primtoflux/vchar and the Lax-Friedrichs flux in float; face
// fluxes stored as float; the flux divergence, flux-CT averaging, the
// connection source, U accumulation, the Noble inversion and the floors in
// double.
#pragma once
#include <cuda_pipeline.h>

#include "harm_common.cuh"
#if HARM_STEP_MIXED
#include "harm_phys32.cuh"
#endif

// Resident blocks of 128 threads per SM that the register allocation must
// allow, per kernel.  The kernels are bound by the latency of dependent FP64
// instructions, so more resident warps beat the few spills the tighter
// register budgets cost; each variant sets values measured best on a B200.
#ifndef HARM_FLUX_MINB
#define HARM_FLUX_MINB 1
#endif
#ifndef HARM_CONS_MINB
#define HARM_CONS_MINB 1
#endif
#ifndef HARM_INV_MINB
#define HARM_INV_MINB 1
#endif

namespace harm {
namespace HARM_VARIANT {

#if HARM_STEP_MIXED
using flux_t = float;
#else
using flux_t = double;
#endif


// faces of direction DIR per theta row and rows per phi plane (step_ch.c:407)
template <int DIR>
__host__ __device__ __forceinline__ int faces_per_row(const Grid &G) { return DIR == 2 ? G.n2 + 1 : G.n2 + 2; }
template <int DIR>
__host__ __device__ __forceinline__ int face_rows(const Grid &G) { return DIR == 1 ? G.n1 + 1 : G.n1 + 2; }

// The face fluxes of every direction in one launch.  Face ranges
// (step_ch.c:407): dir 1 i in [istart, istop+1], j in [jstart-1, jstop+1]; dir 2
// i in [istart-1, istop+1], j in [jstart, jstop+1] (the polar faces jstart and
// jstop+1 carry no flux, :412-416); dir 3 i in [istart-1, istop+1], j in
// [jstart-1, jstop+1].
//
// A block holds FLUX_FACES faces of one direction and phi plane, numbered row
// by row (theta fastest), so that only the plane's last warps have idle lanes.
// Two threads share a face: the first half of the block evaluates the left
// sides, the second half the right sides of the same faces.  They hand each
// other half of their fluxes and conserved variables through shared memory, and
// each forms and stores four of the face's eight fluxes.  The four zones of a
// face's stencil and its metric are copied to shared memory asynchronously, all
// at once, so that a warp waits for one round trip to L2.
//
// What bounds it: issue slots and the latency of dependent FP64 instructions.
// One thread per face held both sides (300 B of spills a thread at 72 registers),
// waited for its loads a few at a time (5.9 of 13.1 warps per issue stalled on
// memory) and issued on half of the cycles; in this form 2.7 stall on memory and
// it issues on 0.62 (FP64) and 0.79 (mixed) of them.  192x192x64, the three
// directions: FP64 825 -> 699 us (the split alone, without the staging, 893),
// mixed 447 -> 428; 288x256x256 FP64 6.77 -> 5.62 ms; 128x128 (launch included)
// 27.7 -> 14.2 us.  64 and 56 registers (8 and 9 blocks) spill again: 756, 810 us.
// With div_rn's shorter last step 663 us (FP64), and with the limiter selected instead
// of branched 623 and 406; 80 registers (6 blocks) 637.
constexpr int FLUX_FACES = 64;

#if HARM_STEP_MIXED
using face_t = float;
using face_geo = GeoF;
#else
using face_t = double;
using face_geo = Geo;
#endif

// the metric entries a face of direction DIR reads, as planes of geo (load_geo's order)
constexpr int FLUX_NG = HARM_STEP_MIXED ? 12 : 14;
template <int DIR>
__device__ constexpr int face_plane(int e)
{
  // v00 v01 v03 v11 v13 v22 v33, n00 n01 n03, n^{dir dir}, g, alpha, 1/alpha
  return e < 10 ? e : e == 10 ? (DIR == 1 ? 11 : DIR == 2 ? 13 : 16) : e + 6;
}

struct FluxShared {
  union {
    double p[8][4][FLUX_FACES];      // primitives of zone-2d, zone-d, zone, zone+d of each face
    face_t x[10][2 * FLUX_FACES];    // four fluxes, four conserved variables, the two wave speeds
  };
  face_t g[FLUX_NG][FLUX_FACES];
  int fail[2 * FLUX_FACES];
  double red[4];
};

// one block's faces of direction DIR; returns this thread's Courant limit.
// REC (the discrete adjoint's recomputation): also keep the wave speed of every
// face that takes part in the Courant minimum, in ctrec[(DIR - 1) nc + cell].
template <int DIR, bool FULL, bool REC>
__device__ __forceinline__ double flux_block(const Grid &G, int fb, int h, const double *__restrict__ pb,
                                             flux_t *__restrict__ F, const face_t *__restrict__ geo, DevScalars *sc,
                                             double *__restrict__ ctrec, FluxShared &S)
{
  const int t = threadIdx.x, side = t / FLUX_FACES, s = t % FLUX_FACES;
  const int nj = faces_per_row<DIR>(G);
  const int f = fb * FLUX_FACES + s;
  const int j = (DIR == 2 ? G.jstart : G.jstart - 1) + f % nj;
  const int i = (DIR == 1 ? G.istart : G.istart - 1) + f / nj;
  const bool in = i <= G.istop + 1;
  const bool pole = DIR == 2 && (j == G.jstart || j == G.jstop + 1);
  const bool calc = in && !pole;
  const long c = cidx(G, h, i, j);
  if (calc) {
    // this thread brings two of the face's four zones and half of its metric
    long o1, o2;
    if (DIR == 1) { o1 = c + (2 * side - 2) * (long)G.sn2; o2 = o1 + G.sn2; }
    else if (DIR == 2) { o1 = c + 2 * side - 2; o2 = o1 + 1; }
    else {
      o1 = cidx(G, hwrap(G, h + 2 * side - 2), i, j);
      o2 = cidx(G, hwrap(G, h + 2 * side - 1), i, j);
    }
#pragma unroll
    for (int k = 0; k < 8; k++) {
      __pipeline_memcpy_async(&S.p[k][2 * side][s], pb + k * G.nc + o1, 8);
      __pipeline_memcpy_async(&S.p[k][2 * side + 1][s], pb + k * G.nc + o2, 8);
    }
    const face_t *gp = geo + (long)(DIR - 1) * GEO_N * G.ng + (long)i * G.sn2 + j;
    if (side == 0) {
#pragma unroll
      for (int e = 0; e < FLUX_NG / 2; e++)
        __pipeline_memcpy_async(&S.g[e][s], gp + face_plane<DIR>(e) * G.ng, sizeof(face_t));
    } else {
#pragma unroll
      for (int e = FLUX_NG / 2; e < FLUX_NG; e++)
        __pipeline_memcpy_async(&S.g[e][s], gp + face_plane<DIR>(e) * G.ng, sizeof(face_t));
    }
  }
  __pipeline_commit();
  __pipeline_wait_prior(0);
  __syncthreads();
  face_t Fs[8], Us[8], cx, cn;
  face_t p[8];
  if (calc) {
    const face_t half = side ? (face_t)-0.5 : (face_t)0.5;
    auto states = [&](int lim) {
#pragma unroll
      for (int k = 0; k < 8; k++) {
        const face_t a = (face_t)S.p[k][side][s], b = (face_t)S.p[k][side + 1][s], e = (face_t)S.p[k][side + 2][s];
#if HARM_STEP_MIXED
        p[k] = b + half * slope_lim_f(lim, a, b, e);
#else
        p[k] = b + half * slope_lim(lim, a, b, e);
#endif
      }
    };
    if (G.lim == 0) states(0);  // one test for the eight, not one each
    else states(G.lim);
  }
  __syncthreads();  // the stencil's space takes the exchange
  if (calc) {
    face_geo q;
    q.v00 = S.g[0][s]; q.v01 = S.g[1][s]; q.v03 = S.g[2][s]; q.v11 = S.g[3][s]; q.v13 = S.g[4][s];
    q.v22 = S.g[5][s]; q.v33 = S.g[6][s];
    q.n00 = S.g[7][s]; q.n01 = S.g[8][s]; q.n03 = S.g[9][s];
    if (DIR == 1) q.n11 = S.g[10][s];
    else if (DIR == 2) q.n22 = S.g[10][s];
    else q.n33 = S.g[10][s];
    q.g = S.g[11][s];
    int fail = 0;
#if HARM_STEP_MIXED
    face_side_f<DIR>((float)G.gam, p, q, Fs, Us, cx, cn, &fail);
#else
    q.alpha = S.g[12][s];
    q.ialpha = S.g[13][s];
    face_side<DIR>(G.gam, p, q, Fs, Us, cx, cn, &fail);
#endif
    if (side == 0) {
#pragma unroll
      for (int k = 0; k < 4; k++) { S.x[k][t] = Fs[4 + k]; S.x[4 + k][t] = Us[4 + k]; }
    } else {
#pragma unroll
      for (int k = 0; k < 4; k++) { S.x[k][t] = Fs[k]; S.x[4 + k][t] = Us[k]; }
    }
    S.x[8][t] = cx;
    S.x[9][t] = cn;
    S.fail[t] = fail;
  }
  __syncthreads();
  double dtmin = 1.e9;
  if (in && pole) {
#pragma unroll
    for (int k = 0; k < 4; k++) F[(4 * side + k) * G.nc + c] = 0.;
  } else if (in) {
    const int o = t ^ FLUX_FACES;  // the face's other side
    const face_t ox = S.x[8][o], on = S.x[9][o];
    const face_t ctop = side == 0 ? lf_speed(cx, cn, ox, on) : lf_speed(ox, on, cx, cn);
    if (side == 0) {
#pragma unroll
      for (int k = 0; k < 4; k++)
        F[k * G.nc + c] = (face_t)0.5 * (Fs[k] + S.x[k][o] - ctop * (S.x[4 + k][o] - Us[k]));
      // the code the sides leave, the right one's last
      const int fail = S.fail[o] ? S.fail[o] : S.fail[t];
      if (fail) record_fail(sc, fail, h + (G.n3 > 1 ? 1 : 0), i, j);
      if (FULL && i >= G.istart && i <= G.istop && j >= G.jstart && j <= G.jstop) {
        const double dxd = DIR == 1 ? G.dx1 : DIR == 2 ? G.dx2 : G.dx3;
        dtmin = G.cour * dxd / (double)ctop;
        if (REC && DIR < 3) ctrec[(DIR - 1) * G.nc + c] = (double)ctop;
      }
    } else {
#pragma unroll
      for (int k = 0; k < 4; k++)
        F[(4 + k) * G.nc + c] = (face_t)0.5 * (S.x[k][o] + Fs[4 + k] - ctop * (Us[4 + k] - S.x[4 + k][o]));
    }
  }
  return dtmin;
}

// blocks per phi plane of each direction
struct FluxBlocks {
  int b1, b2, b3;
};

template <bool FULL, bool REC, bool THREE_D>
__global__ void __launch_bounds__(2 * FLUX_FACES, HARM_FLUX_MINB) k_flux(Grid G, FluxBlocks nb,
                                                                         const double *__restrict__ pb,
                                                                         flux_t *__restrict__ F1,
                                                                         flux_t *__restrict__ F2,
                                                                         flux_t *__restrict__ F3,
                                                                         const face_t *__restrict__ geo,
                                                                         DevScalars *sc, double *__restrict__ ctrec)
{
  if (sc->halted) return;
  __shared__ FluxShared S;
  if (blockIdx.x == 0 && threadIdx.x == 0) sc->nfail[FULL ? 1 : 0] = 0;  // for this half step's repairs
  int b = blockIdx.x, dir;
  double dtmin;
  if (b < nb.b1 * G.n3) {
    dir = 1;
    dtmin = flux_block<1, FULL, REC>(G, b % nb.b1, b / nb.b1, pb, F1, geo, sc, ctrec, S);
  } else if (!THREE_D || (b -= nb.b1 * G.n3) < nb.b2 * G.n3) {
    if (!THREE_D) b -= nb.b1;
    dir = 2;
    dtmin = flux_block<2, FULL, REC>(G, b % nb.b2, b / nb.b2, pb, F2, geo, sc, ctrec, S);
  } else {
    b -= nb.b2 * G.n3;
    dir = 3;
    dtmin = flux_block<3, FULL, REC>(G, b % nb.b3, b / nb.b3, pb, F3, geo, sc, ctrec, S);
  }
  if (FULL) {
    const int t = threadIdx.x;
    double v = warp_min(dtmin);
    if ((t & 31) == 0) S.red[t >> 5] = v;
    __syncthreads();
    if (t == 0) {
      v = fmin(fmin(S.red[0], S.red[1]), fmin(S.red[2], S.red[3]));
      if (v < 1.e9) atomicMin(&sc->ndt_bits[dir - 1], (unsigned long long)__double_as_longlong(v));
    }
  }
}

// ctrec (the adjoint's recomputation of a corrector): keep the direction-1
// and -2 faces' wave speeds there
template <bool FULL>
void launch_flux(const Grid &G, cudaStream_t st, const double *pb, flux_t *F1, flux_t *F2, flux_t *F3,
                 const double *geo64, const float *geo32, DevScalars *sc, double *ctrec = nullptr)
{
#if HARM_STEP_MIXED
  const float *geo = geo32;
#else
  const double *geo = geo64;
#endif
  auto blocks = [](int faces) { return (faces + FLUX_FACES - 1) / FLUX_FACES; };
  const FluxBlocks nb{blocks(faces_per_row<1>(G) * face_rows<1>(G)), blocks(faces_per_row<2>(G) * face_rows<2>(G)),
                      G.n3 > 1 ? blocks(faces_per_row<3>(G) * face_rows<3>(G)) : 0};
  const unsigned grid = (unsigned)(nb.b1 + nb.b2 + nb.b3) * G.n3;
  const int nt = 2 * FLUX_FACES;
#if !HARM_STEP_MIXED
  if (FULL && ctrec) {
    // ctrec holds directions 1 and 2 (the adjoint that reads it is 2D); a 3D
    // step still gets its phi fluxes, without a record
    if (G.n3 > 1) k_flux<true, true, true><<<grid, nt, 0, st>>>(G, nb, pb, F1, F2, F3, geo, sc, ctrec);
    else k_flux<true, true, false><<<grid, nt, 0, st>>>(G, nb, pb, F1, F2, F3, geo, sc, ctrec);
    return;
  }
#endif
  if (G.n3 > 1) k_flux<FULL, false, true><<<grid, nt, 0, st>>>(G, nb, pb, F1, F2, F3, geo, sc, nullptr);
  else k_flux<FULL, false, false><<<grid, nt, 0, st>>>(G, nb, pb, F1, F2, F3, geo, sc, nullptr);
}

// ---------------------------------------------------------------------------
// update (step_ch.c:237-306) fused with flux_ct (step_ch.c:514-629, 726-798),
// the flux boundary fixes (coord.c:264-324) and fixup() (fixup.c:51-60)

struct Flux {
  const flux_t *F1, *F2, *F3;
  Grid G;
  __device__ double raw(int d, int k, int h, int i, int j) const
  {
    const flux_t *F = d == 1 ? F1 : d == 2 ? F2 : F3;
    return (double)__ldg(F + k * G.nc + cidx(G, h, i, j));
  }
  // B-component of a raw face flux after fix_flux's polar reflection
  // (coord.c:284-301): F1,F3[B2] at jstart-1 / jstop+1 mirror jstart / jstop
  __device__ double rawB2(int d, int h, int i, int j) const
  {
    if (j == G.jstart - 1) return -raw(d, B2, h, i, G.jstart);
    if (j == G.jstop + 1) return -raw(d, B2, h, i, G.jstop);
    return raw(d, B2, h, i, j);
  }
  // 2D EMF (step_ch.c:546-547)
  __device__ double emf2(int i, int j) const
  {
    return 0.25 * (rawB2(1, 0, i, j) + rawB2(1, 0, i, j - 1) - raw(2, B1, 0, i, j) - raw(2, B1, 0, i - 1, j));
  }
  // 3D EMFs (step_ch.c:754-764); h-1 wraps (phi periodic)
  __device__ double e1(int h, int i, int j) const
  {
    int hm = hwrap(G, h - 1);
    return 0.25 * ((raw(2, B3, h, i, j) + raw(2, B3, hm, i, j)) - (rawB2(3, h, i, j) + rawB2(3, h, i, j - 1)));
  }
  __device__ double e2(int h, int i, int j) const
  {
    int hm = hwrap(G, h - 1);
    return 0.25 * ((raw(3, B1, h, i, j) + raw(3, B1, h, i - 1, j)) - (raw(1, B3, h, i, j) + raw(1, B3, hm, i, j)));
  }
  __device__ double e3(int h, int i, int j) const
  {
    return 0.25 * ((rawB2(1, h, i, j) + rawB2(1, h, i, j - 1)) - (raw(2, B1, h, i, j) + raw(2, B1, h, i - 1, j)));
  }
};

template <bool THREE_D>
__device__ void zone_fluxes(const Flux &FX, int h, int i, int j, double *f1m, double *f1p, double *f2m,
                            double *f2p, double *f3m, double *f3p)
{
  const Grid &G = FX.G;
  const int hp = THREE_D ? hwrap(G, h + 1) : 0;
#pragma unroll
  for (int k = 0; k < 5; k++) {
    f1m[k] = FX.raw(1, k, h, i, j);
    f1p[k] = FX.raw(1, k, h, i + 1, j);
    f2m[k] = FX.raw(2, k, h, i, j);
    f2p[k] = FX.raw(2, k, h, i, j + 1);
    if (THREE_D) {
      f3m[k] = FX.raw(3, k, h, i, j);
      f3p[k] = FX.raw(3, k, hp, i, j);
    }
  }
  // no inflow of mass through the radial boundaries (coord.c:307-321)
  if (i == G.istart && f1m[RHO] > 0) f1m[RHO] = 0;
  if (i + 1 == G.istop + 1 && f1p[RHO] < 0) f1p[RHO] = 0;
  if (!THREE_D) {
    double eA = FX.emf2(i, j), eB = FX.emf2(i, j + 1), eC = FX.emf2(i + 1, j), eD = FX.emf2(i + 1, j + 1);
    f1m[B1] = 0.;
    f1m[B2] = 0.5 * (eA + eB);
    f1m[B3] = FX.raw(1, B3, 0, i, j);
    f1p[B1] = 0.;
    f1p[B2] = 0.5 * (eC + eD);
    f1p[B3] = FX.raw(1, B3, 0, i + 1, j);
    f2m[B1] = -0.5 * (eA + eC);
    f2m[B2] = 0.;
    f2m[B3] = FX.raw(2, B3, 0, i, j);
    f2p[B1] = -0.5 * (eB + eD);
    f2p[B2] = 0.;
    f2p[B3] = FX.raw(2, B3, 0, i, j + 1);
  } else {
    double e3a = FX.e3(h, i, j), e3b = FX.e3(h, i, j + 1), e3c = FX.e3(h, i + 1, j), e3d = FX.e3(h, i + 1, j + 1);
    double e2a = FX.e2(h, i, j), e2b = FX.e2(hp, i, j), e2c = FX.e2(h, i + 1, j), e2d = FX.e2(hp, i + 1, j);
    double e1a = FX.e1(h, i, j), e1b = FX.e1(hp, i, j), e1c = FX.e1(h, i, j + 1), e1d = FX.e1(hp, i, j + 1);
    f1m[B1] = 0.;
    f1m[B2] = 0.5 * (e3a + e3b);
    f1m[B3] = -0.5 * (e2a + e2b);
    f1p[B1] = 0.;
    f1p[B2] = 0.5 * (e3c + e3d);
    f1p[B3] = -0.5 * (e2c + e2d);
    f2m[B1] = -0.5 * (e3a + e3c);
    f2m[B2] = 0.;
    f2m[B3] = 0.5 * (e1a + e1b);
    f2p[B1] = -0.5 * (e3b + e3d);
    f2p[B2] = 0.;
    f2p[B3] = 0.5 * (e1c + e1d);
    f3m[B1] = 0.5 * (e2a + e2c);
    f3m[B2] = -0.5 * (e1a + e1c);
    f3m[B3] = 0.;
    f3p[B1] = 0.5 * (e2b + e2d);
    f3p[B2] = -0.5 * (e1b + e1d);
    f3p[B3] = 0.;
  }
}

// flux_ct's corner EMFs (step_ch.c:514-629 in 2D, 726-798 in 3D), each
// formed once from the raw face fluxes, for the update of the four zones that
// share the corner: emf[2 nc + cell] e3 (2D: the one EMF), and in 3D emf[cell]
// e1, emf[nc + cell] e2.  Corners i in [istart, istop+1], j in [jstart,
// jstop+1], every phi plane.
template <bool THREE_D>
__global__ void __launch_bounds__(128) k_emf(Grid G, const flux_t *__restrict__ F1, const flux_t *__restrict__ F2,
                                             const flux_t *__restrict__ F3, double *__restrict__ emf, DevScalars *sc)
{
  if (sc->halted) return;
  const int nj = G.n2 + 1;
  const int f = blockIdx.x * 128 + threadIdx.x;
  const int j = G.jstart + f % nj, i = G.istart + f / nj;
  if (i > G.istop + 1) return;
  const int h = blockIdx.z;
  const Flux FX{F1, F2, F3, G};
  const long c = cidx(G, h, i, j);
  if (THREE_D) {
    emf[c] = FX.e1(h, i, j);
    emf[G.nc + c] = FX.e2(h, i, j);
    emf[2 * G.nc + c] = FX.e3(h, i, j);
  } else {
    emf[2 * G.nc + c] = FX.emf2(i, j);
  }
}

// Where the update takes a corner's EMFs from: the planes k_emf filled, or (2D)
// the raw face fluxes around the corner.
struct EmfPlanes {
  const double *emf;
  __device__ __forceinline__ double at(const Grid &G, int n, int h, int i, int j) const
  {
    return __ldg(emf + n * G.nc + cidx(G, h, i, j));
  }
};
struct EmfFaces {
  const Flux &FX;
  __device__ __forceinline__ double at(const Grid &, int, int, int i, int j) const { return FX.emf2(i, j); }
};

// The flux divergence of the update (step_ch.c:247-263) one conserved
// component at a time, U[k] += Dt (-dF1/dx1 - dF2/dx2 [- dF3/dx3] + dU[k]), with
// the same face fluxes zone_fluxes forms (the no-inflow mass-flux fix, and the
// field components rebuilt from the corner EMFs of flux_ct), so only one
// component's six face values are live at a time.
template <bool THREE_D, class Emf>
__device__ __forceinline__ void flux_update(const Flux &FX, const Emf &emf, int h, int i, int j, double Dt,
                                            const double *dU, double *U)
{
  const Grid &G = FX.G;
  const int hp = THREE_D ? hwrap(G, h + 1) : 0;
  auto upd = [&](int k, double f1m, double f1p, double f2m, double f2p, double f3m, double f3p) {
#if HARM_STEP_MIXED
    const double idx1 = 1. / G.dx1, idx2 = 1. / G.dx2, idx3 = 1. / G.dx3;
    if (THREE_D)
      U[k] += Dt * (-(f1p - f1m) * idx1 - (f2p - f2m) * idx2 - (f3p - f3m) * idx3 + dU[k]);
    else
      U[k] += Dt * (-(f1p - f1m) * idx1 - (f2p - f2m) * idx2 + dU[k]);
#else
    if (THREE_D)
      U[k] += Dt * (-div_rn(f1p - f1m, G.dx1, G.idx1) - div_rn(f2p - f2m, G.dx2, G.idx2)
                    - div_rn(f3p - f3m, G.dx3, G.idx3) + dU[k]);
    else
      U[k] += Dt * (-div_rn(f1p - f1m, G.dx1, G.idx1) - div_rn(f2p - f2m, G.dx2, G.idx2) + dU[k]);
#endif
  };
#pragma unroll
  for (int k = 0; k < 5; k++) {
    double f1m = FX.raw(1, k, h, i, j), f1p = FX.raw(1, k, h, i + 1, j);
    if (k == RHO) {
      // no inflow of mass through the radial boundaries (coord.c:307-321)
      if (i == G.istart && f1m > 0) f1m = 0;
      if (i + 1 == G.istop + 1 && f1p < 0) f1p = 0;
    }
    const double f2m = FX.raw(2, k, h, i, j), f2p = FX.raw(2, k, h, i, j + 1);
    const double f3m = THREE_D ? FX.raw(3, k, h, i, j) : 0., f3p = THREE_D ? FX.raw(3, k, hp, i, j) : 0.;
    upd(k, f1m, f1p, f2m, f2p, f3m, f3p);
  }
  if (!THREE_D) {
    const double eA = emf.at(G, 2, 0, i, j), eB = emf.at(G, 2, 0, i, j + 1);
    const double eC = emf.at(G, 2, 0, i + 1, j), eD = emf.at(G, 2, 0, i + 1, j + 1);
    upd(B1, 0., 0., -0.5 * (eA + eC), -0.5 * (eB + eD), 0., 0.);
    upd(B2, 0.5 * (eA + eB), 0.5 * (eC + eD), 0., 0., 0., 0.);
    upd(B3, FX.raw(1, B3, 0, i, j), FX.raw(1, B3, 0, i + 1, j), FX.raw(2, B3, 0, i, j), FX.raw(2, B3, 0, i, j + 1),
        0., 0.);
  } else {
    const double e3a = emf.at(G, 2, h, i, j), e3b = emf.at(G, 2, h, i, j + 1);
    const double e3c = emf.at(G, 2, h, i + 1, j), e3d = emf.at(G, 2, h, i + 1, j + 1);
    const double e2a = emf.at(G, 1, h, i, j), e2b = emf.at(G, 1, hp, i, j);
    const double e2c = emf.at(G, 1, h, i + 1, j), e2d = emf.at(G, 1, hp, i + 1, j);
    upd(B1, 0., 0., -0.5 * (e3a + e3c), -0.5 * (e3b + e3d), 0.5 * (e2a + e2c), 0.5 * (e2b + e2d));
    const double e1a = emf.at(G, 0, h, i, j), e1b = emf.at(G, 0, hp, i, j);
    const double e1c = emf.at(G, 0, h, i, j + 1), e1d = emf.at(G, 0, hp, i, j + 1);
    upd(B2, 0.5 * (e3a + e3b), 0.5 * (e3c + e3d), 0., 0., -0.5 * (e1a + e1c), -0.5 * (e1b + e1d));
    upd(B3, -0.5 * (e2a + e2b), -0.5 * (e2c + e2d), 0.5 * (e1a + e1b), 0.5 * (e1c + e1d), 0., 0.);
  }
}

// What the update of a zone reads besides the state and the fluxes.
struct ZoneData {
  const double *geo, *conn;
  const float *geo32, *conn32;
  const double *floors, *katm;
};

// A block's zones in shared memory: 32 points of the (r, theta) grid, numbered row by
// row, on PL phi planes.  The points' metric and connection are shared by the
// planes; everything comes in one round trip to L2, asynchronously.
template <bool FULL, int PL>
struct ZoneShared {
  double conn[40][32];           // (mixed, away from the horizon: floats, in the slots' low halves)
  double geo[GEO_N][32];
  double pb[8][PL][32];
  double pi[FULL ? 8 : 1][PL][32];  // the predictor advances from pi == pb
#if HARM_STEP_MIXED
  float geo32[11][32];
#endif
};

// Where the update takes a zone's operands from: the staged block (3D), or the planes
// in memory (2D, where no other plane shares a point's 61 metric and connection
// entries and staging them only delays the first use: 128x128 update 28.4 us
// staged, 25.6 direct).
struct ConnShared {
  const double *c;  // the point's first entry
  __device__ __forceinline__ double operator()(int slot) const { return c[slot * 32]; }
};
template <bool FULL, int PL>
struct StagedZone {
  const ZoneShared<FULL, PL> &S;
  __device__ __forceinline__ double pb(int k) const { return S.pb[k][threadIdx.y][threadIdx.x]; }
  __device__ __forceinline__ double pi(int k) const { return FULL ? S.pi[k][threadIdx.y][threadIdx.x] : pb(k); }
  __device__ __forceinline__ ConnShared conn() const { return ConnShared{&S.conn[0][threadIdx.x]}; }
  __device__ __forceinline__ void geo(Geo &q) const
  {
    const int x = threadIdx.x;
    q.v00 = S.geo[0][x]; q.v01 = S.geo[1][x]; q.v03 = S.geo[2][x]; q.v11 = S.geo[3][x]; q.v13 = S.geo[4][x];
    q.v22 = S.geo[5][x]; q.v33 = S.geo[6][x];
    q.n00 = S.geo[7][x]; q.n01 = S.geo[8][x]; q.n03 = S.geo[9][x]; q.n10 = S.geo[10][x]; q.n11 = S.geo[11][x];
    q.n13 = S.geo[12][x]; q.n22 = S.geo[13][x]; q.n30 = S.geo[14][x]; q.n31 = S.geo[15][x]; q.n33 = S.geo[16][x];
    q.g = S.geo[17][x];
    q.alpha = S.geo[18][x]; q.ialpha = S.geo[19][x]; q.ig = S.geo[20][x];
  }
#if HARM_STEP_MIXED
  struct Conn32 {
    const double *c;
    __device__ __forceinline__ float operator()(int slot) const
    {
      return *reinterpret_cast<const float *>(c + slot * 32);
    }
  };
  __device__ __forceinline__ Conn32 conn32() const { return Conn32{&S.conn[0][threadIdx.x]}; }
  __device__ __forceinline__ void geo32(GeoF &q) const
  {
    const int x = threadIdx.x;
    q.v00 = S.geo32[0][x]; q.v01 = S.geo32[1][x]; q.v03 = S.geo32[2][x]; q.v11 = S.geo32[3][x];
    q.v13 = S.geo32[4][x]; q.v22 = S.geo32[5][x]; q.v33 = S.geo32[6][x];
    q.n00 = S.geo32[7][x]; q.n01 = S.geo32[8][x]; q.n03 = S.geo32[9][x];
    q.g = S.geo32[10][x];
  }
#endif
};
struct DirectZone {
  const Grid &G;
  const double *ppi, *ppb;
  const ZoneData &Z;
  long c, gi;
  __device__ __forceinline__ double pb(int k) const { return __ldg(ppb + k * G.nc + c); }
  __device__ __forceinline__ double pi(int k) const { return ppi[k * G.nc + c]; }
  __device__ __forceinline__ ConnPlanes conn() const { return ConnPlanes{Z.conn + gi, G.ng}; }
  __device__ __forceinline__ void geo(Geo &q) const { load_geo(geo_at(Z.geo, G, L_CENT), G.ng, gi, q); }
#if HARM_STEP_MIXED
  struct Conn32 {
    const float *conn;
    long ng;
    __device__ __forceinline__ float operator()(int slot) const { return __ldg(conn + slot * ng); }
  };
  __device__ __forceinline__ Conn32 conn32() const { return Conn32{Z.conn32 + gi, G.ng}; }
  __device__ __forceinline__ void geo32(GeoF &q) const
  {
    load_geo_f(Z.geo32 + (long)L_CENT * GEO_N * G.ng, G.ng, gi, q);
  }
#endif
};
#if HARM_STEP_MIXED
// the entries of a point's FP32 metric that the source reads, as planes of geo32
__device__ constexpr int source_plane(int e) { return e < 10 ? e : 17; }
#endif

// ok: the point is in the grid; in_plane: and so is this thread's plane
template <bool FULL, int PL>
__device__ __forceinline__ void stage_zone(const Grid &G, ZoneShared<FULL, PL> &S, const double *pi, const double *pb,
                                           const ZoneData &Z, bool ok, bool in_plane, int h, int i, int j)
{
  const int x = threadIdx.x, y = threadIdx.y;
  if (ok) {
    const long gi = (long)i * G.sn2 + j;
    const double *g = Z.geo + (long)L_CENT * GEO_N * G.ng + gi;
#pragma unroll
    for (int e = 0; e < GEO_N; e += PL)
      if (e + y < GEO_N) __pipeline_memcpy_async(&S.geo[e + y][x], g + (e + y) * G.ng, 8);
#if HARM_STEP_MIXED
    if (i >= G.isrc32) {
      const float *c = Z.conn32 + gi, *f = Z.geo32 + (long)L_CENT * GEO_N * G.ng + gi;
#pragma unroll
      for (int e = 0; e < 40; e += PL) __pipeline_memcpy_async(&S.conn[e + y][x], c + (e + y) * G.ng, 4);
#pragma unroll
      for (int e = 0; e < 11; e += PL)
        if (e + y < 11) __pipeline_memcpy_async(&S.geo32[e + y][x], f + source_plane(e + y) * G.ng, 4);
    } else
#endif
    {
      const double *c = Z.conn + gi;
#pragma unroll
      for (int e = 0; e < 40; e += PL) __pipeline_memcpy_async(&S.conn[e + y][x], c + (e + y) * G.ng, 8);
    }
    if (in_plane) {
      const long c = cidx(G, h, i, j);
#pragma unroll
      for (int k = 0; k < 8; k++) {
        __pipeline_memcpy_async(&S.pb[k][y][x], pb + k * G.nc + c, 8);
        if (FULL) __pipeline_memcpy_async(&S.pi[k][y][x], pi + k * G.nc + c, 8);
      }
    }
  }
  __pipeline_commit();
  __pipeline_wait_prior(0);
  __syncthreads();
}

// U of zone (h, i, j) after the half step: flux_ct (step_ch.c:514-629,
// 726-798), the flux boundary fixes (coord.c:264-324), source() (phys.c:165-207),
// primtoU of pi and the flux divergence (step_ch.c:247-263).  The order of every
// floating-point operation is the reference's.
template <bool FULL, bool THREE_D, class Zone, class Emf>
__device__ __forceinline__ void cons_zone(const Grid &G, const Zone &zone, const Flux &FX, const Emf &emf,
                                          const Geo &q, double Dt, int h, int i, int j, double *U, int *fail)
{
  double dU[8];
  double pz[8];
#if HARM_STEP_MIXED
  if (i >= G.isrc32) {
    // away from the horizon: the connection source in float (harm_phys32.cuh)
    float pf32[8];
#pragma unroll
    for (int k = 0; k < 8; k++) pf32[k] = (float)zone.pb(k);
    GeoF qf;
    zone.geo32(qf);
    source_f((float)G.gam, pf32, qf, zone.conn32(), dU, fail);
#pragma unroll
    for (int k = 0; k < 8; k++) pz[k] = zone.pi(k);
    State s;
    get_state(pz, q, s, fail);
    primtoflux(G.gam, pz, s, 0, q.g, U);
  } else
#endif
  {
    State s;
#pragma unroll
    for (int k = 0; k < 8; k++) pz[k] = zone.pb(k);
    get_state(pz, q, s, fail);
    source_of_state(G.gam, pz, s, q, zone.conn(), dU);
    if (FULL) {
#pragma unroll
      for (int k = 0; k < 8; k++) pz[k] = zone.pi(k);
      get_state(pz, q, s, fail);
    }  // the predictor (advance(p, p, ...), step_ch.c:101): one state serves both
    primtoflux(G.gam, pz, s, 0, q.g, U);
  }
  flux_update<THREE_D>(FX, emf, h, i, j, Dt, dU, U);
}

// The block of the update's first half: 32 points of the grid on four phi planes in
// 3D, 128 points in 2D, numbered row by row.
constexpr int ZONE_PLANES = 4;
template <bool THREE_D>
__device__ __forceinline__ bool zone_of_thread(const Grid &G, int &h, int &i, int &j)
{
  const int z = blockIdx.x * blockDim.x + threadIdx.x;
  j = G.jstart + z % G.n2;
  i = G.istart + z / G.n2;
  h = THREE_D ? blockIdx.z * ZONE_PLANES + threadIdx.y : 0;
  return i <= G.istop;
}

// Large grids take the update in two launches, so that each holds fewer
// registers and more warps stay resident to cover FP64 latency: k_cons forms U
// into Ub, k_invert inverts it.
//
// k_cons in 3D is bound by the latency of its loads: when each thread loaded its
// zone's 61 metric and connection entries as it used them, 7.4 of 13 warps per issue
// waited on memory.  Staged, once for four planes: update of 192x192x64 FP64 692 ->
// 654 us, 288x256x256 5.54 -> 5.36 ms, 70x50x22 55 -> 49 us.
template <bool FULL, bool THREE_D>
__global__ void __launch_bounds__(128, HARM_CONS_MINB) k_cons(Grid G, const double *__restrict__ pi,
                                                              const double *__restrict__ pb,
                                                              const flux_t *__restrict__ F1,
                                                              const flux_t *__restrict__ F2,
                                                              const flux_t *__restrict__ F3, ZoneData Z,
                                                              const double *__restrict__ emf,
                                                              double *__restrict__ Ub, DevScalars *sc)
{
  if (sc->halted) return;
  int h, i, j, fail = 0;
  const bool ok = zone_of_thread<THREE_D>(G, h, i, j), in = ok && h < G.n3;
  const double Dt = FULL ? sc->dt : 0.5 * sc->dt;
  const long c = cidx(G, h, i, j);
  const Flux FX{F1, F2, F3, G};
  Geo q;
  double U[8];
  if (THREE_D) {
    __shared__ ZoneShared<FULL, ZONE_PLANES> S;
    stage_zone<FULL, ZONE_PLANES>(G, S, pi, pb, Z, ok, in, h, i, j);
    if (!in) return;
    const StagedZone<FULL, ZONE_PLANES> zone{S};
    zone.geo(q);
    cons_zone<FULL, THREE_D>(G, zone, FX, EmfPlanes{emf}, q, Dt, h, i, j, U, &fail);
  } else {
    if (!in) return;
    const DirectZone zone{G, pi, pb, Z, c, (long)i * G.sn2 + j};
    zone.geo(q);
    cons_zone<FULL, THREE_D>(G, zone, FX, EmfPlanes{emf}, q, Dt, h, i, j, U, &fail);
  }
#pragma unroll
  for (int k = 0; k < 8; k++) Ub[k * G.nc + c] = U[k];
  if (fail) record_fail(sc, fail, h + (THREE_D ? 1 : 0), i, j);
}

// the isentropic fall-backs (step_ch.c:277-300), kept out of line: most
// zones never take them, and inlined they crowd the kernel's hot code out of
// the instruction cache; which: 1 or 2, the last one tried
static __device__ __noinline__ int inversion_fallbacks(double gam, double kap, const double *U, const Geo &q,
                                                       double *pz, int *which)
{
  int flag = utoprim<1>(gam, kap, U, q, pz);
  *which = 1;
  if (flag) {
    flag = utoprim<2>(gam, kap, U, q, pz);
    *which = 2;
  }
  return flag;
}

// What a half step does with a zone's inverted primitives.
struct ZoneOut {
  double *pf;
  signed char *pflag;   // 1 a good zone, 0 a failed one: as fixup_utoprim leaves the flags
  int *list;            // failed zones, listed for the repair
  double *zrec;         // (the adjoint) the inversion's output before fixup()
  signed char *wrec;    // and which inversion gave it
};

// bound_prim()'s copies of an edge zone of a 2D grid (bounds.c:54-378): every
// ghost cell there is made from one active zone, the two next to a radial
// boundary from the edge zone (then inflow_check), the two next to a pole by
// reflection.  The zone's own thread writes them.
static __device__ __noinline__ void push_ghosts(const Grid &G, const ZoneOut &O, const double *__restrict__ geo,
                                                DevScalars *sc, int i, int j, const double *v, signed char fl)
{
  const int jm = j == G.jstart ? j - 1 : j == G.jstart + 1 ? j - 3 : j == G.jstop ? j + 1 : j == G.jstop - 1 ? j + 3 : -1;
  const int n = i == G.istart || i == G.istop ? 3 : 1;
  for (int m = 0; m < 2; m++) {
    const int jt = m ? jm : j;
    if (jt < 0) continue;
    for (int r = 0; r < n; r++) {
      const int it = i == G.istart ? i - r : i + r;
      if (m == 0 && r == 0) continue;
      double w[8];
#pragma unroll
      for (int k = 0; k < 8; k++) w[k] = v[k];
      if (m) {
        w[U2] *= -1.;
        w[B2] *= -1.;
      }
      const long gi = (long)it * G.sn2 + jt;
      if (r) {
        Geo q;
        load_geo(geo_at(geo, G, L_CENT), G.ng, gi, q);
        int fail = 0;
        inflow_check(w, q, i == G.istart ? 0 : 1, &fail);
        if (fail) record_fail(sc, fail, 0, it, jt);
      }
#pragma unroll
      for (int k = 0; k < 8; k++) O.pf[k * G.nc + gi] = w[k];
      O.pflag[gi] = fl;
    }
  }
}

// Utoprim_2d with the isentropic fall-backs (step_ch.c:265-300) and fixup()
// (fixup.c:142-383) of one zone; pz holds the guess (pi).  REC: also keep the
// inversion's output before fixup() and which inversion gave it, for the discrete
// adjoint's recomputation.  PUSH (2D, in the one-launch update): write the zone's ghost
// cells too.
template <bool REC, bool PUSH>
__device__ __forceinline__ void invert_zone(const Grid &G, const double *U, const Geo &q, double *pz,
                                            const ZoneData &Z, const ZoneOut &O, DevScalars *sc, int slot, int h,
                                            int i, int j)
{
  const long c = cidx(G, h, i, j);
  const long gi = (long)i * G.sn2 + j;
  int fail = 0;
  int flag = utoprim<0, (bool)HARM_STEP_MIXED>(G.gam, 0., U, q, pz);
  int which = 0;
  if (flag) {
    // on copies made here: arrays whose address a call takes would live in memory for
    // the whole kernel, the Newton solve's operands among them
    double Uc[8], pc[8];
    const Geo qc = q;
    int w;
#pragma unroll
    for (int k = 0; k < 8; k++) { Uc[k] = U[k]; pc[k] = pz[k]; }
    flag = inversion_fallbacks(G.gam, __ldg(Z.katm + i), Uc, qc, pc, &w);
#pragma unroll
    for (int k = 0; k < 8; k++) pz[k] = pc[k];
    which = w;
  }
  if (REC) {
#pragma unroll
    for (int k = 0; k < 8; k++) O.zrec[k * G.nc + c] = pz[k];
    O.wrec[c] = (signed char)(flag ? -1 : which);
  }
  signed char fl = (signed char)flag;
  if (fixup1zone(G.gam, __ldg(Z.floors + gi), __ldg(Z.floors + G.ng + gi), q, pz, &fail)) fl = -33;
  // fixup_utoprim's flip of the flags (fixup.c:432-445), and its list
  fl = (signed char)(!fl);
  if (fl == 0) list_failed(sc, slot, O.list, c);
#pragma unroll
  for (int k = 0; k < 8; k++) O.pf[k * G.nc + c] = pz[k];
  O.pflag[c] = fl;
  if (PUSH && (i == G.istart || i == G.istop || j <= G.jstart + 1 || j >= G.jstop - 1)) {
    double v[8];
#pragma unroll
    for (int k = 0; k < 8; k++) v[k] = pz[k];
    push_ghosts(G, O, Z.geo, sc, i, j, v, fl);
  }
  if (fail) record_fail(sc, fail, h + (G.n3 > 1 ? 1 : 0), i, j);
}

template <bool REC>
__global__ void __launch_bounds__(128, HARM_INV_MINB) k_invert(Grid G, const double *__restrict__ pi,
                                                               const double *__restrict__ Ub, ZoneData Z, ZoneOut O,
                                                               int slot, int hb, DevScalars *sc)
{
  if (sc->halted) return;
  const int j = G.jstart + blockIdx.x * blockDim.x + threadIdx.x;
  const int i = G.istart + blockIdx.y * blockDim.y + threadIdx.y;
  if (i > G.istop || j > G.jstop) return;
  const int h0 = blockIdx.z * hb, h1 = min(G.n3, h0 + hb);
  for (int h = h0; h < h1; h++) {
    const long c = cidx(G, h, i, j);
    Geo q;
    load_geo(geo_at(Z.geo, G, L_CENT), G.ng, (long)i * G.sn2 + j, q);
    double U[8], pz[8];
#pragma unroll
    for (int k = 0; k < 8; k++) {
      U[k] = __ldg(Ub + k * G.nc + c);
      pz[k] = pi[k * G.nc + c];
    }
    invert_zone<REC, false>(G, U, q, pz, Z, O, sc, slot, h, i, j);
  }
}

// Small grids take the whole update in one launch, zones numbered row by row: each
// launch of a step costs them some 2 us beside the latency of its loads.  With the
// ghosts, flags and failure list written here, the sums and the dt update in one
// launch and the repair with its bound_prim in another, a 2D step is 7 launches
// instead of 22: 128x128 FP64 85.8 -> 69 us, 251x187 mixed 87 -> 71 us.
template <bool FULL, bool THREE_D, bool REC>
__global__ void __launch_bounds__(128, UPD_MINB) k_update(Grid G, const double *pi, const double *pb,
                                                               const flux_t *__restrict__ F1,
                                                               const flux_t *__restrict__ F2,
                                                               const flux_t *__restrict__ F3, ZoneData Z,
                                                               const double *__restrict__ emf, ZoneOut O,
                                                               double *__restrict__ Ub, DevScalars *sc)
{
  if (sc->halted) return;
  int h, i, j, fail = 0;
  const bool ok = zone_of_thread<THREE_D>(G, h, i, j), in = ok && h < G.n3;
  const double Dt = FULL ? sc->dt : 0.5 * sc->dt;
  const long c = cidx(G, h, i, j);
  const Flux FX{F1, F2, F3, G};
  Geo q;
  double U[8], pz[8];
  if (THREE_D) {
    __shared__ ZoneShared<FULL, ZONE_PLANES> S;
    stage_zone<FULL, ZONE_PLANES>(G, S, pi, pb, Z, ok, in, h, i, j);
    if (!in) return;
    const StagedZone<FULL, ZONE_PLANES> zone{S};
    zone.geo(q);
    cons_zone<FULL, THREE_D>(G, zone, FX, EmfPlanes{emf}, q, Dt, h, i, j, U, &fail);
#pragma unroll
    for (int k = 0; k < 8; k++) pz[k] = zone.pi(k);
  } else {
    if (!in) return;
    const DirectZone zone{G, pi, pb, Z, c, (long)i * G.sn2 + j};
    zone.geo(q);
    cons_zone<FULL, THREE_D>(G, zone, FX, EmfFaces{FX}, q, Dt, h, i, j, U, &fail);
#pragma unroll
    for (int k = 0; k < 8; k++) pz[k] = zone.pi(k);
  }
  if (fail) record_fail(sc, fail, h + (THREE_D ? 1 : 0), i, j);
  if (REC) {
#pragma unroll
    for (int k = 0; k < 8; k++) Ub[k * G.nc + c] = U[k];
  }
  invert_zone<REC, !THREE_D>(G, U, q, pz, Z, O, sc, FULL ? 1 : 0, h, i, j);
}

// ---------------------------------------------------------------------------
// one step of this variant

struct Bufs {
  flux_t *F1, *F2, *F3;
};

inline Bufs bufs(Ctx *x)
{
#if HARM_STEP_MIXED
  return Bufs{x->F1f, x->F2f, x->F3f};
#else
  return Bufs{x->F1, x->F2, x->F3};
#endif
}

// Ub, zrec, wrec: the adjoint's recomputation keeps U, the inversion's output and
// which inversion gave it there
template <bool FULL>
void launch_update(Ctx *x, const double *pi, const double *pb, double *pf, double *Ub = nullptr,
                   double *zrec = nullptr, signed char *wrec = nullptr)
{
  const Grid &G = x->G;
  Bufs B = bufs(x);
  const ZoneData Z{x->geo, x->conn, x->geo32, x->conn32, x->floors, x->katm};
  const ZoneOut O{pf, x->pflag, x->fail_list, zrec, wrec};
  const long zones = (long)G.n1 * G.n2 * G.n3;
  const bool fused = fused_update(G);
  const dim3 eg(((G.n2 + 1) * (G.n1 + 1) + 127) / 128, 1, G.n3);
  if (G.n3 > 1) k_emf<true><<<eg, 128, 0, x->stream>>>(G, B.F1, B.F2, B.F3, x->emf, x->sc);
  else if (!fused) k_emf<false><<<eg, 128, 0, x->stream>>>(G, B.F1, B.F2, B.F3, x->emf, x->sc);
  const dim3 cb = G.n3 > 1 ? dim3(32, ZONE_PLANES) : dim3(128);
  const dim3 cg((G.n1 * G.n2 + cb.x - 1) / cb.x, 1, (G.n3 + ZONE_PLANES - 1) / ZONE_PLANES);
  if (fused) {
    if (G.n3 > 1)
      k_update<FULL, true, false><<<cg, cb, 0, x->stream>>>(G, pi, pb, B.F1, B.F2, B.F3, Z, x->emf, O, nullptr, x->sc);
#if !HARM_STEP_MIXED
    else if (zrec)
      k_update<FULL, false, true><<<cg, cb, 0, x->stream>>>(G, pi, pb, B.F1, B.F2, B.F3, Z, x->emf, O, Ub, x->sc);
#endif
    else
      k_update<FULL, false, false><<<cg, cb, 0, x->stream>>>(G, pi, pb, B.F1, B.F2, B.F3, Z, x->emf, O, nullptr, x->sc);
    return;
  }
  // phi planes a block of k_invert sweeps: four, whose zones share the tile's geometry in L1,
  // where that still leaves eight blocks for every SM, one where it does not
  // (70x50x22: update 82 us with four, 55 with one)
  const int hb = zones >= 148L * 8 * 128 * 4 ? 4 : 1;
  const dim3 tile(x->tbx, x->tby);
  const dim3 zg((G.n2 + tile.x - 1) / tile.x, (G.n1 + tile.y - 1) / tile.y, (G.n3 + hb - 1) / hb);
  double *U = Ub ? Ub : x->Ubuf;
  if (G.n3 > 1) k_cons<FULL, true><<<cg, cb, 0, x->stream>>>(G, pi, pb, B.F1, B.F2, B.F3, Z, x->emf, U, x->sc);
  else k_cons<FULL, false><<<cg, cb, 0, x->stream>>>(G, pi, pb, B.F1, B.F2, B.F3, Z, x->emf, U, x->sc);
#if !HARM_STEP_MIXED
  if (zrec) {
    k_invert<true><<<zg, tile, 0, x->stream>>>(G, pi, U, Z, O, FULL ? 1 : 0, hb, x->sc);
    return;
  }
#endif
  k_invert<false><<<zg, tile, 0, x->stream>>>(G, pi, U, Z, O, FULL ? 1 : 0, hb, x->sc);
}

// advance() + fixup + bound_prim + fixup_utoprim + bound_prim (step_ch.c:101-117);
// a 2D update in one launch writes the ghosts
template <bool FULL>
void launch_half(Ctx *x, const double *pi, const double *pb, double *pf)
{
  Bufs B = bufs(x);
  launch_flux<FULL>(x->G, x->stream, pb, B.F1, B.F2, B.F3, x->geo, x->geo32, x->sc);
  launch_update<FULL>(x, pi, pb, pf);
  if (!update_writes_ghosts(x->G)) launch_bound(x, pf);
  launch_repair(x, pf, FULL ? 1 : 0);
}

int launch_step(Ctx *x)
{
  launch_half<false>(x, x->p, x->p, x->ph);
  launch_half<true>(x, x->p, x->ph, x->p);
  launch_mass(x, bufs(x).F1);
  CK(cudaGetLastError());
  return HARM_OK;
}

#if !HARM_STEP_MIXED
// launch_half and launch_step as above, also keeping what the discrete adjoint
// reads back (StepRec); the same kernels in the same order, so the recomputed
// step is the step (2D)
template <bool FULL>
static int launch_half_rec(Ctx *x, const double *pi, const double *pb, double *pf, const StepRec &r)
{
  const int s = FULL ? 1 : 0;
  const size_t nc = (size_t)x->G.nc;
  Bufs B = bufs(x);
  launch_flux<FULL>(x->G, x->stream, pb, B.F1, B.F2, B.F3, x->geo, x->geo32, x->sc, FULL ? r.ctop : nullptr);
  CK(cudaMemcpyAsync(r.F1rho[s], B.F1 + RHO * nc, nc * sizeof(double), cudaMemcpyDeviceToDevice, x->stream));
  launch_update<FULL>(x, pi, pb, pf, r.Ub[s], r.Z[s], r.wz[s]);
  if (!update_writes_ghosts(x->G)) launch_bound(x, pf);
  CK(cudaMemcpyAsync(r.X1[s], pf, 8 * nc * sizeof(double), cudaMemcpyDeviceToDevice, x->stream));
  CK(cudaMemcpyAsync(r.fl1[s], x->pflag, nc, cudaMemcpyDeviceToDevice, x->stream));
  CK(cudaMemcpyAsync(r.nfail[s], &x->sc->nfail[s], sizeof(int), cudaMemcpyDeviceToDevice, x->stream));
  return launch_repair(x, pf, s);
}

int launch_step_rec(Ctx *x, const StepRec &r)
{
  int rc = launch_half_rec<false>(x, x->p, x->p, x->ph, r);
  if (rc) return rc;
  cudaMemcpyAsync(r.ph, x->ph, 8 * (size_t)x->G.nc * sizeof(double), cudaMemcpyDeviceToDevice, x->stream);
  rc = launch_half_rec<true>(x, x->p, x->ph, x->p, r);
  if (rc) return rc;
  // the corrector's Courant minima, before k_mass resets them
  cudaMemcpyAsync(r.sc[0], x->sc, sizeof(DevScalars), cudaMemcpyDeviceToDevice, x->stream);
  launch_mass(x, bufs(x).F1);
  cudaMemcpyAsync(r.sc[1], x->sc, sizeof(DevScalars), cudaMemcpyDeviceToDevice, x->stream);
  CK(cudaGetLastError());
  return HARM_OK;
}
#endif

// reps ordinary steps, one kernel at a time with an event after each, so
// every kernel is timed inside the sequence it runs in; slots: flux, update,
// bound_prim (where the update does not write the ghosts), fixup_utoprim with the
// bound_prim after it, diagnostics
int time_kernels(Ctx *x, int reps, double *ms)
{
  const Grid &G = x->G;
  Bufs B = bufs(x);
  const int nev = 16;
  cudaEvent_t ev[nev];
  for (auto &e : ev) CK(cudaEventCreate(&e));
  double acc[HARM_NKERNELS] = {0, 0, 0, 0, 0};
  for (int r = 0; r < reps; r++) {
    int e = 0, slot[nev];
    CK(cudaEventRecord(ev[e++], x->stream));
    for (int half = 0; half < 2; half++) {
      const bool full = half == 1;
      double *pi = x->p, *pb = full ? x->ph : x->p, *pf = full ? x->p : x->ph;
      if (full) launch_flux<true>(G, x->stream, pb, B.F1, B.F2, B.F3, x->geo, x->geo32, x->sc);
      else launch_flux<false>(G, x->stream, pb, B.F1, B.F2, B.F3, x->geo, x->geo32, x->sc);
      slot[e] = 0; CK(cudaEventRecord(ev[e++], x->stream));
      if (full) launch_update<true>(x, pi, pb, pf);
      else launch_update<false>(x, pi, pb, pf);
      slot[e] = 1; CK(cudaEventRecord(ev[e++], x->stream));
      if (!update_writes_ghosts(G)) {
        launch_bound(x, pf);
        slot[e] = 2; CK(cudaEventRecord(ev[e++], x->stream));
      }
      launch_repair(x, pf, half);
      slot[e] = 3; CK(cudaEventRecord(ev[e++], x->stream));
    }
    launch_mass(x, B.F1);
    slot[e] = 4; CK(cudaEventRecord(ev[e++], x->stream));
    CK(cudaEventSynchronize(ev[e - 1]));
    for (int k = 1; k < e; k++) {
      float f;
      CK(cudaEventElapsedTime(&f, ev[k - 1], ev[k]));
      acc[slot[k]] += f;
    }
  }
  for (auto &e : ev) cudaEventDestroy(e);
  const double per_step[HARM_NKERNELS] = {2, 2, 2, 2, 1};
  for (int k = 0; k < HARM_NKERNELS; k++) ms[k] = acc[k] / (reps * per_step[k]);
  return sync_status(x);
}

}  // namespace HARM_VARIANT
}  // namespace harm

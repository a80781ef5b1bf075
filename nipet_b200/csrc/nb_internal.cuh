// nb_internal.cuh -- geometry handle layout and host-side helpers shared by the
// translation units of libnipet_b200.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>

#include "nb_common.cuh"

// Per-ray description, canonical ray order r in [0, 4084):
//   r <  64           direct plane of ring li = r
//   r <  64 + 2010    oblique +RD ray of ring pair li = r                (ring r0 -> r1)
//   r <  4084         oblique -RD ray of ring pair li = r - 2010         (ring r1 -> r0)
// (the reference's fprj_oblq computes the +RD and -RD rays of a pair in one thread).
struct nb_ray {
  float r0z, r1z;     // li2rng[li] (ring front edges, cm)
  int16_t out11;      // span-11 sinogram of the ray
  int16_t out1;       // span-1 sinogram of the ray
  int8_t kind;        // 0 direct, 1 +RD, 2 -RD
  int8_t nos;         // span-1 planes in its span-11 sinogram (li2nos)
  int16_t li;
};

// A ray pair of the projector kernels (one per thread and turn): ring pair (r0, r0 + d) with
// its upward ray A (r0 -> r1) and downward ray B (r1 -> r0), or for d = 0 two direct planes.
// Slots are ordered by d, so the lanes of a warp make about equally many plane crossings.
struct nb_slot {
  uint32_t zzd;        // plane of ring r0 (2 r0) | plane of ring r1 << 8 | d << 16 (direct: the
                       // two planes)
  int16_t o11A, o11B;  // span-11 sinogram of each ray, -1: no such ray
  int16_t o1A, o1B;    // span-1 sinogram (a reduced range's own numbers in nb_rings)
  int16_t nosA, nosB;  // span-1 planes in the ray's span-11 sinogram
};
#define NB_NSLOT 2048  // slot table capacity: 32 for the direct planes, 2010 pairs, padding

// Crossing schedule of a LOR (k_sched, nb_geom.cu), 16-byte aligned.  Schedule d is that of the
// ring pairs of difference d; 61 .. 63 are those of pairs that cross at other floats than the
// rest of their difference.
//   kend[52][64]  crossings of a schedule up to and including the steps of 8-step row r
//   m[64]         first plane boundary the upward ray crosses, relative to its ring's 2 r0
//   off[64]       first entry of a schedule (uint16)
//   meta          uint16 count of irregular rays, then the differences of schedules 61 .. 63
//   irr[96]       {d, r0, 0 up / 1 down, start plane offset}: rays whose start plane rounds
//                 away from their schedule's; {d, r0, 2, schedule}: pairs that follow another
//   entries       {int32 step, int32 fraction of the step before the crossing (2^26 = 1)}
#define NB_REC_KEND 0
#define NB_REC_M 3328
#define NB_REC_OFF 3392
#define NB_REC_META 3520
#define NB_REC_IRR 3536
#define NB_REC_MAXIRR 96
#define NB_REC_NALT 3
#define NB_REC_ENT 3920
#define NB_REC_MAXENT 3584
#define NB_REC_QBITS 26
#define NB_REC_MAX (NB_REC_ENT + 8 * NB_REC_MAXENT)

struct nb_geom {
  int device;
  int nsm;
  int naw;
  // Siddon step lists: [naw][NB_STEP_STRIDE]
  int32_t *d_scol;   // transaxial column (v*320 + u) of each step
  float *d_st;       // exit parameter t of each step (the entry is the previous exit)
  float4 *d_hdr;     // per LOR: (t entry of step 0, atn, t2, nsteps as int bits)
  float *d_tt;       // reference-layout tt [naw][10]
  nb_ray *d_rays;    // [4084]
  unsigned char *d_rec;  // crossing schedules of all LORs
  uint32_t *d_rec_off;   // [naw + 1] start of a LOR's record, in 16-byte units
  nb_slot *d_slots;      // [nslots] ray pairs
  int nslots;        // 0: rays that are not the mMR's ring pairs, or whose crossings do not fit the
                     // schedules; every projection runs step by step over d_rays (k_walk_any)
  int16_t *d_bin11;  // [837][8] rays of each span-11 sinogram (-1 padded): 2 slot + direction, or
                     // the index in d_rays without slots
  float *d_scratch128;   // one col128 image (reference-layout entry points)
  int *d_err;            // device error flag
  float *d_one;          // the constant 1.0f (randoms factor of a single-image batch)
  // host copies of the LUTs (for nb_geom_tables) and of the ray table (for nb_rings_create)
  float h_crs[504 * 4];
  int16_t *h_s2c;
  nb_ray *h_rays;    // [4084], as d_rays
};

// The rays of a reduced axial ring range [rs, re) (span 1 only): the reference's
// Cnt.RNG_STRT / RNG_END mode, in which projections cover the ring pairs inside the range,
// sinograms are numbered by the range's own span-1 Michelogram and images hold the axial
// voxel slab [vz0, vz0 + nvz) with nvz = 2 (re - rs) - 1 (prj/src/prjf.cu:209-320,
// prjb.cu:190-308, mmraux.py:566-617).  Every ray is one of the geometry's own rays, so
// the walk checks of nb_geom_create cover it.
struct nb_rings {
  int device;
  int rs, re;
  int nrays;         // rays of the range = its span-1 sinograms
  int vz0, nvz;
  nb_slot *d_slots;  // [nslots] the range's ray pairs, o1A / o1B the range's sinograms
  int nslots;        // 0: step by step over d_rays
  nb_ray *d_rays;    // [nrays]
};

// ---- tracing: an NVTX range around a C-ABI call (header-only NVTX3: without a profiler
// attached a push / pop costs a branch) ----
#include <nvtx3/nvToolsExt.h>
struct NbRange {
  explicit NbRange(const char *name) { nvtxRangePushA(name); }
  ~NbRange() { nvtxRangePop(); }
  NbRange(const NbRange &) = delete;
  NbRange &operator=(const NbRange &) = delete;
};
#define NB_RANGE(name) NbRange nb_range_(name)

// ---- host-side error plumbing (nb_capi.cu) ----
void nb_set_error_msg(const char *fmt, ...);
int nb_cuda_fail(cudaError_t e, const char *what, const char *file, int line);

#define NB_CUDA(call)                                                                          \
  do {                                                                                         \
    cudaError_t _e = (call);                                                                   \
    if (_e != cudaSuccess) return nb_cuda_fail(_e, #call, __FILE__, __LINE__);                 \
  } while (0)

#define NB_REQUIRE(cond, msg)                                                                  \
  do {                                                                                         \
    if (!(cond)) {                                                                             \
      nb_set_error_msg("%s", msg);                                                             \
      return NB_ERR_ARG;                                                                       \
    }                                                                                          \
  } while (0)

// multiprocessors of the current device
static inline int nb_sms() {
  int dev = 0, nsm = 148;
  if (cudaGetDevice(&dev) == cudaSuccess)
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  return nsm;
}

// Check the device error flag of a handle after synchronising `stream` (debug/validation
// paths only; the hot entry points do not synchronise).
int nb_check_device_flag(nb_geom *g, cudaStream_t stream);

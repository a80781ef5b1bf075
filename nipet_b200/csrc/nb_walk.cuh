// nb_walk.cuh -- the projector kernel: forward projection, back projection and the fused
// OSEM sub-iteration of BS images at a time (BS = 1, 2 or 4), used by nb_prj.cu and
// nb_batch.cu.
//
// Reference semantics: prj/src/prjf.cu:33-206 (fprj_drct, fprj_oblq), prj/src/prjb.cu:33-187
// (bprj_drct, bprj_oblq), prj/src/recon.cu:252-309 and :459-497 (OSEM sub-iteration).
//
// The walk.  A LOR (transaxial sinogram bin) crosses n ~ 270 voxel columns; its 4084 rays
// (ring pairs, both directions) share those steps and differ in the axial plane they are
// in.  A ray changes plane only ~35 times, so instead of visiting a voxel per step
// (n reads a ray) the kernel forms, per plane z, the running integral C_i[z] of the columns
// over the steps, and a ray needs one interpolated difference D[P] = C[P-1] - C[P] at each
// of its crossings of a plane boundary P, plus C at the plane it ends in:
//     ray = sum over crossings +-( D_i[P] + f * lt_i * (x_i[P-1] - x_i[P]) ) + C_end[z_end]
// (a crossing in step i at the fraction f of the step).  The back projection is the adjoint:
// a crossing moves a ray's value V from plane to plane, (1 - f) V in step i and f V in step
// i + 1, and a running sum over the steps turns these flows into what each plane receives.
//
// The schedule.  Rays of one ring difference d and both directions cross planes at the
// same steps and fractions, 2 planes apart per ring, so the crossings of a LOR are one list
// per d (~3000 entries for all 4084 rays), made once per geometry (nb_geom.cu: k_sched) and
// streamed into shared memory with the LOR (24 KB, one bulk copy).
//
// Exactness.  Running integrals are int32 fixed point, one power-of-two scale per chunk of
// CH steps and image (2^29 over a bound of the planes' integrals of |value|, so that the
// difference of two planes of opposite sign fits as well), so the differences cancel exactly: a
// ray through empty planes is exactly zero whatever its neighbours hold, and integer sums do not
// depend on the order.  A ray's own sum, with the fraction terms, is 64 bits wide: it collects
// from one plane after another and can exceed what any of them holds.
//   The scale is set by the chunk's hottest plane, so a ray through values decades below it is a
// sum of few quanta.  At the end of a LOR, rays below 2^20 quanta per chunk whose planes hold weak
// values, and any below 1.5 x 2^16, are walked again step by step in float32, as the reference
// walks every ray (walk_weak); so are all rays of an image whose chunk has no scale (a value that
// is not finite, or above 2^100).  The fused mode leaves out those whose ratio does not need them:
// nothing counted, or randoms above 2^20 quanta.  Every bin is then good to 1e-5 of its value, but
// for slivers of a step (a fraction is good to 2^-25 of the step).
//   In the back projection a ray's value is rounded once, by at most 2^-23 of the LOR's largest,
// and its two parts of a crossing sum to it exactly.  The weights that meet in a plane in one step
// sum to 255 at the most (checked when the geometry is made: a late crossing has weights outside
// [0, 1]) and values are below 2^23, so no sum leaves int32.  An image with a value that is not finite goes to the voxels ray by ray in float32.
//
// Jobs.  One block per (LOR, image group); a finished block takes over a block that has not
// started (cluster launch control), so LORs of 10 to 404 steps even out over the SMs and the
// next LOR's copies are in flight while one ends (a fixed stride over the LORs left the last
// wave 9% of the SMs' time idle at 4894 LORs).
//
// Measured (B200, 1965 MHz; per call, against the step-by-step walk it replaces): attenuation
// factors of all LORs at span 11 28.0 -> 3.3 ms (chunks without any value are skipped), a
// 4894-LOR emission projection 2.16 -> 0.29 ms, a 5003-LOR span-1 back projection 2.57 ->
// 0.84 ms, a drop-in OSEM iteration 64.4 -> 20.4 ms, 9 images batched 341 -> 161 ms.  Against
// the FP64 oracle the error is less than half (forward 1.1e-7 -> 5e-8, back 1.7e-7 -> 6e-8
// relative L2).  An image with 1e-5 around an object in place of zeros, whose weak rays (1000 on a
// LOR through the object) are walked again, takes 1.12 ms for 4894 LORs in place of 0.68.
// What bounds it: the shared-memory (LSU) pipe at 70 (forward) to 79% of its wavefronts for one
// image, half of them the crossings' (a warp of 32 pairs spans up to 8 ring differences, whose lanes
// share banks: 3.1 wavefronts per 8-byte read where 2 would do); of the time the crossings take
// a third, the running sums a fifth, each chunk's set-up of the pairs a seventh, the rest loads,
// bounds and the LOR's start and end.  Aligning differences to half-warps saved 20% of the
// crossings' wavefronts and lost more to 20% more sets (0.77 -> 0.85 ms); warps that own steps
// instead (no tables: one shared reduction per crossing and ray) took 1.5 to 2 times as long
// for one image and as long for four.
#pragma once
#include "nb_axial.cuh"
#include "nb_internal.cuh"

namespace nbw {

constexpr uint32_t WAIT_POLLS = 1u << 20;
enum { MODE_FWD = 0, MODE_BWD = 1, MODE_OSEM = 2 };
constexpr int FXBITS = 23;    // back projection: |V| <= 2^23 (see the file comment)
// A ray's sum is good to float32's precision from so many quanta per chunk on: a ray through
// weak values, whose every voxel is rounded; and any other, which may clip a voxel or two
constexpr float WEAK_QUANTA = 1048576.f, CLIP_QUANTA = 98304.f;   // 2^20, 1.5 * 2^16
// A value is weak below 2^15 quanta for a step of 1/16 cm
constexpr float WEAK_VALUE = 524288.f;
constexpr int QBITS = NB_REC_QBITS;  // crossing fractions are int32 with this many fraction bits

struct WalkArgs {
  const int32_t *scol;
  const float *st;
  const float4 *hdr;
  const unsigned char *rec;   // crossing schedules (nb_internal.cuh: NB_REC_*)
  const uint32_t *rec_off;    // [naw + 1] start of a LOR's record, in 16-byte units
  const nb_slot *slots;
  int nslots;
  const nb_ray *rays;         // [nrays], for k_walk_any (nslots 0)
  int nrays;
  const int16_t *bin11;       // [837][8] rays (2 * slot + direction) of each span-11 sinogram
  const int32_t *subs;
  int nprj, naw, ngroups, nrep;
  int nout;                   // sinograms per row (837, 4084, or a reduced range's count)
  int span;                   // 1 or 11
  int att;                    // forward: 0 emission, 1 attenuation factors
  int in_by_lor;              // backward: row of a LOR is its LOR index, not its subset position
  const float *img;           // [ngroups][NCOL][128][BS]
  int natural;                // forward, BS 1: img is the reference's [NCOL][127] instead
  float *bimg;                // same layout, accumulated
  float *sino;                // forward output [nrep][nprj][nout]
  const float *sino_in;       // backward input [nrep][nprj][nout] (or [naw][nout] if in_by_lor)
  const uint16_t *psng;       // OSEM prompts [nrep][naw][nout]
  const float *rs;            // OSEM (r+s)/(an) [naw][nout], scaled per image by rscale
  const float *rscale;        // [nrep]
  int *err;
};

__host__ __device__ constexpr size_t align128(size_t x) { return (x + 127) & ~(size_t)127; }
__host__ __device__ constexpr size_t cmax(size_t a, size_t b) { return a > b ? a : b; }

// Shared memory.  The forward tables (per step 128 planes of {D, dX} per image), the span-11
// ray values and the backward accumulators with their float staging are never live
// together and share one region.
template <int BS, int CH, int NSEG> struct WSmem {
  static constexpr size_t tab = (size_t)CH * 1024 * BS;
  static constexpr size_t gacc = (size_t)(CH + 1) * 512 * BS;
  static_assert(gacc >= 4096ull * 4 * BS, "a LOR's ray values fit the accumulators");
  static constexpr size_t stage = (size_t)CH * 512 * BS;
  static constexpr size_t region = cmax(cmax(tab, 4096ull * 4 * BS), align128(gacc) + stage);
  static constexpr size_t stg_off = align128(gacc);
  static constexpr size_t seg_off = align128(region);                       // [NSEG][128][BS]
  static constexpr size_t oc_off = align128(seg_off + 512ull * NSEG * BS);  // [NSEG][steps + 1][BS]
  static constexpr size_t run_off = align128(oc_off + 4ull * (CH + NSEG) * BS);      // [2][128][BS]
  static constexpr size_t rec_off = align128(run_off + 1024ull * BS);
  static constexpr size_t cs_off = align128(rec_off + NB_REC_MAX);          // [2][2][stride]
  static constexpr size_t max_off = align128(cs_off + 16ull * NB_STEP_STRIDE);  // [3][NSEG][BS]
  static constexpr size_t obl_off = align128(max_off + 12ull * NSEG * BS);      // [64]
  static constexpr size_t misc_off = obl_off + 256;
  static constexpr size_t total = misc_off + 256;
  // walk_weak: the rays' integrals [4096][BS], the list of rays, then columns of the image
  static constexpr size_t list_off = 4096ull * 4 * BS;
  static constexpr size_t col_off = list_off + 4096 * 2;
  static constexpr int ncol = (int)((region - col_off) / (512 * BS)) & ~7;
  static_assert(region >= col_off + 16 * 512 * BS, "room for some columns");
  static_assert(total <= 227 * 1024, "too much shared memory");
};

template <int N> struct VecF;
template <> struct VecF<1> { using T = float; };
template <> struct VecF<2> { using T = float2; };
template <> struct VecF<4> { using T = float4; };
template <int N> struct VecI;
template <> struct VecI<1> { using T = int; };
template <> struct VecI<2> { using T = int2; };
template <> struct VecI<4> { using T = int4; };

template <int N> __device__ __forceinline__ void ldv(const float *p, float *v) {
  const typename VecF<N>::T t = *reinterpret_cast<const typename VecF<N>::T *>(p);
  const float *q = reinterpret_cast<const float *>(&t);
#pragma unroll
  for (int k = 0; k < N; k++) v[k] = q[k];
}
template <int N> __device__ __forceinline__ void ldg_v(const float *p, float *v) {
  const typename VecF<N>::T t = __ldg(reinterpret_cast<const typename VecF<N>::T *>(p));
  const float *q = reinterpret_cast<const float *>(&t);
#pragma unroll
  for (int k = 0; k < N; k++) v[k] = q[k];
}
template <int N> __device__ __forceinline__ void ldi(const int *p, int *v) {
  const typename VecI<N>::T t = *reinterpret_cast<const typename VecI<N>::T *>(p);
  const int *q = reinterpret_cast<const int *>(&t);
#pragma unroll
  for (int k = 0; k < N; k++) v[k] = q[k];
}
template <int N> __device__ __forceinline__ void sti(int *p, const int *v) {
  typename VecI<N>::T t;
  int *q = reinterpret_cast<int *>(&t);
#pragma unroll
  for (int k = 0; k < N; k++) q[k] = v[k];
  *reinterpret_cast<typename VecI<N>::T *>(p) = t;
}

// shared-memory accessors on 32-bit shared-window addresses
static __device__ __forceinline__ void lds_ent(uint32_t addr, int &i, int &f) {
  asm volatile("ld.shared.v2.b32 {%0,%1}, [%2];" : "=r"(i), "=r"(f) : "r"(addr));
}
static __device__ __forceinline__ void reds_add_s32(uint32_t addr, int v) {
  asm volatile("red.shared.add.s32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}
// {D, dD} of BS images at a table address: 8 bytes (BS 1), 16 (BS 2: D0 D1 dD0 dD1), or two
// 16-byte rows 2 KB apart (BS 4), so that the lanes of a warp read consecutive banks
template <int BS>
static __device__ __forceinline__ void lds_tab(uint32_t addr, int *D, int *X) {
  if (BS == 1) {
    asm volatile("ld.shared.v2.b32 {%0,%1}, [%2];" : "=r"(D[0]), "=r"(X[0]) : "r"(addr));
  } else if (BS == 2) {
    asm volatile("ld.shared.v4.b32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(D[0]), "=r"(D[1]), "=r"(X[0]), "=r"(X[1])
                 : "r"(addr));
  } else {
    asm volatile("ld.shared.v4.b32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(D[0]), "=r"(D[1]), "=r"(D[2]), "=r"(D[3])
                 : "r"(addr));
    asm volatile("ld.shared.v4.b32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(X[0]), "=r"(X[1]), "=r"(X[2]), "=r"(X[3])
                 : "r"(addr + 2048u));
  }
}

// byte offset of a plane in a row whose planes are `unit` bytes wide (even planes first)
static __device__ __forceinline__ int plane_off(int P, int unit) {
  return P * (unit / 2) + (P & 1) * (127 * unit / 2);
}
// u + x / 2^QBITS as float32: the words one by one (exactly 0 for 0; a small negative sum is off
// by 2^-18 at the most)
static __device__ __forceinline__ float quanta(int u, long long x) {
  x += (long long)u * (1 << QBITS);
  return fmaf((float)(int)(x >> 32), (float)(1 << (32 - QBITS)),
              (float)(uint32_t)x * (1.f / (1 << QBITS)));
}
static __device__ __forceinline__ float oblique_s(int d, float atn) {
  if (d == 0) return 1.f;
  const float az_atn = __fdiv_rn((float)d * NB_RING, atn);
  return __fsqrt_rn(__fmaf_rn(az_atn, az_atn, 1.0f));
}

// does [lo, hi] hold a plane of the mask (words: planes 0, 2 .. 62; 64 .. 126; 1 .. 63; 65 .. 127)
static __device__ __forceinline__ bool mask_meets(const unsigned *mask, int lo, int hi) {
  bool hit = false;
#pragma unroll
  for (int par = 0; par < 2; par++) {
    const uint2 m2 = *reinterpret_cast<const uint2 *>(mask + 2 * par);
    const unsigned long long m = (unsigned long long)m2.y << 32 | m2.x;
    const int a = (lo + 1 - par) >> 1, b = (hi - par) >> 1;   // b = -1: no odd plane below 1
    hit |= b >= a && (m >> a & (~0ull >> (63 - (b - a)))) != 0ull;
  }
  return hit;
}

// A ray of the slots as the reference's axial set-up sees it
static __device__ __forceinline__ void slot_axial(const nb_slot *slots, int ray, const float4 &h,
                                                  nb_axial &A) {
  const uint32_t zz = slots[ray >> 1].zzd;
  const int d = (int)(zz >> 16);
  nb_axial_setup(nb_ring_pair((int)((d ? zz : zz >> (ray & 1) * 8) & 255u) / 2, d,
                              d ? 1 + (ray & 1) : 0), h.y, h.x, h.z, A);
}

// Up to NT / 8 rays of `list` step by step in float32, straight from the image: a ray in 8 to 32
// parts, whose lanes find their start by the crossings alone.  (Staged as below they would wait
// for five rounds of copies: 33 LORs, which take 22 us, took 30 us longer.)  Sums are formed per
// block of 8 steps and added up in order, as there: a ray's result depends on neither the number
// of rays nor the lanes.  sums: NB_STEP_STRIDE / 8 blocks a ray.
template <int BS, int NT>
static __device__ __noinline__ void walk_few(const float *gimg, size_t stride, bool natural,
                                             const int32_t *scol, const float *sst, int n,
                                             const float4 h, const nb_slot *slots,
                                             const uint16_t *list, int count, float *vals,
                                             float *sums) {
  constexpr int U = 4;                        // steps whose reads are in flight together
  const int tid = threadIdx.x;
  const int lanes = count <= NT / 32 ? 32 : (count <= NT / 16 ? 16 : 8), sub = tid & (lanes - 1);
  const bool live = tid / lanes < count;
  const int ray = list[live ? tid / lanes : 0], part = ((n + lanes - 1) / lanes + 7) & ~7;
  const int s0 = min(n, sub * part), s1 = live ? min(n, s0 + part) : 0;
  nb_axial A;
  slot_axial(slots, ray, h, A);
  int z = A.w;
  float tp = h.x, tzc = A.tzc, acc[BS];
  if (s0 < s1 && s0 > 0) {
    // the crossings before the last four steps (s0 is a multiple of four), then those steps one
    // by one: a crossing put off to the next step has caught up by then
    const float t0 = s0 > 4 ? sst[s0 - 5] : h.x;
    for (int c = 0; c < s0 - 4 && t0 > tzc; c++) {
      z += A.dir;
      tzc = __fadd_rn(tzc, A.dtz);
    }
    float t[4];
    ldv<4>(sst + s0 - 4, t);
#pragma unroll
    for (int u = 0; u < 4; u++)
      if (t[u] > tzc) {
        z += A.dir;
        tzc = __fadd_rn(tzc, A.dtz);
      }
    tp = t[3];
  }
  float *mine = sums + (size_t)(tid / lanes) * (NB_STEP_STRIDE / 8) * BS;
  for (int s = s0; s < s1; s += U) {
    if ((s & 7) == 0)
#pragma unroll
      for (int k = 0; k < BS; k++) acc[k] = 0.f;
    float v0[U][BS], v1[U][BS], w0[U], w1[U];
#pragma unroll
    for (int u = 0; u < U; u++) {
      w0[u] = w1[u] = 0.f;
#pragma unroll
      for (int k = 0; k < BS; k++) v0[u][k] = v1[u][k] = 0.f;
      if (s + u >= s1) continue;
      const float tn = sst[s + u];
      const float *c = gimg + (size_t)scol[s + u] * stride;
      if (!natural || z < NB_IMZ) ldg_v<BS>(c + (natural ? z : nb_zi(z) * BS), v0[u]);
      w0[u] = __fsub_rn(fminf(tn, tzc), tp);
      if (tn > tzc) {
        z += A.dir;
        if (!natural || z < NB_IMZ) ldg_v<BS>(c + (natural ? z : nb_zi(z) * BS), v1[u]);
        w1[u] = __fsub_rn(tn, tzc);
        tzc = __fadd_rn(tzc, A.dtz);
      }
      tp = tn;
    }
#pragma unroll
    for (int u = 0; u < U; u++)
#pragma unroll
      for (int k = 0; k < BS; k++) acc[k] = fmaf(w1[u], v1[u][k], fmaf(w0[u], v0[u][k], acc[k]));
    if ((s & 4) || s + U >= s1)
#pragma unroll
      for (int k = 0; k < BS; k++) mine[(s >> 3) * BS + k] = acc[k];
  }
  __syncwarp();
  if (live && sub == 0) {
#pragma unroll
    for (int k = 0; k < BS; k++) acc[k] = 0.f;
    for (int b = 0; b < (n + 7) / 8; b++)
#pragma unroll
      for (int k = 0; k < BS; k++) acc[k] += mine[b * BS + k];
#pragma unroll
    for (int k = 0; k < BS; k++) vals[ray * BS + k] = acc[k];
  }
}

// Fused mode: has the LOR a bin whose ratio could need more than 2^20 quanta per chunk?  Not where
// nothing was counted, nor where the randoms outweigh them.  (Asked for the bins in order, before
// the rays: late iterates of noisy data have weak rays on every LOR and no such bin.)
template <int BS, int NT>
static __device__ __noinline__ bool bins_matter(const WalkArgs &a, const float *sthr, int g, int lor) {
  bool some = false;
  const size_t row = (size_t)lor * a.nout;
  const float *rs = a.rs + row;
  const uint16_t *y[BS];
  float lim[BS], scale[BS];
#pragma unroll
  for (int k = 0; k < BS; k++) {
    const int rep = min(g * BS + k, a.nrep - 1);   // (a padding image repeats the last one)
    y[k] = a.psng + (size_t)rep * a.naw * a.nout + row;
    scale[k] = a.rscale[rep];
    lim[k] = sthr[k] * WEAK_QUANTA;
    some |= lim[k] == __int_as_float(0x7f800000);
  }
  // four bins at a time where rows allow it (span 1)
  const bool vec = a.nout % 4 == 0 && (((uintptr_t)a.rs & 15) | ((uintptr_t)a.psng & 7)) == 0;
  if (vec) {
#pragma unroll 2
    for (int o = threadIdx.x; o < a.nout / 4; o += NT) {
      const float4 r = __ldg(reinterpret_cast<const float4 *>(rs) + o);
#pragma unroll
      for (int k = 0; k < BS; k++) {
        const ushort4 c = __ldg(reinterpret_cast<const ushort4 *>(y[k]) + o);
        some |= ((c.x != 0) & !(scale[k] * r.x >= lim[k])) | ((c.y != 0) & !(scale[k] * r.y >= lim[k])) |
                ((c.z != 0) & !(scale[k] * r.z >= lim[k])) | ((c.w != 0) & !(scale[k] * r.w >= lim[k]));
      }
    }
  } else {
#pragma unroll 2
    for (int o = threadIdx.x; o < a.nout; o += NT) {
      const float r = __ldg(rs + o);
#pragma unroll
      for (int k = 0; k < BS; k++) some |= (__ldg(y[k] + o) != 0) & !(scale[k] * r >= lim[k]);
    }
  }
  return some;
}

// Walks the rays of a LOR whose fixed-point sums (vals, [4096][BS]) are too few quanta to be good
// to float32's precision again: step by step in float32, as the reference does, from columns
// staged in shared memory (40 KB at a time).  All threads; false if there was none to walk.
template <int BS, int NT, int MODE, class L>
static __device__ __noinline__ bool walk_weak(const WalkArgs &a, unsigned char *smem, int par,
                                              int g, int lor, int n, const float4 h) {
  static_assert(NT % (128 * BS) == 0, "a thread stays with its plane and image");
  const int32_t *scol = reinterpret_cast<const int32_t *>(
      smem + L::cs_off + (size_t)par * 8 * NB_STEP_STRIDE);
  const float *sst = reinterpret_cast<const float *>(scol) + NB_STEP_STRIDE;
  const unsigned char *rec = smem + L::rec_off;
  float *vals = reinterpret_cast<float *>(smem);
  uint16_t *list = reinterpret_cast<uint16_t *>(smem + L::list_off);
  float *cols = reinterpret_cast<float *>(smem + L::col_off);
  unsigned char *misc = smem + L::misc_off;
  int *scount = reinterpret_cast<int *>(misc + 40);
  const float *sthr = reinterpret_cast<const float *>(misc + 96);
  const int *sweak = reinterpret_cast<const int *>(misc + 112);
  unsigned *smask = reinterpret_cast<unsigned *>(misc + 176);   // [BS][4] planes of weak values
  const int tid = threadIdx.x;
  const bool natural = MODE == MODE_FWD && BS == 1 && a.natural != 0;
  const size_t stride = natural ? NB_IMZ : NB_COLW * BS;
  const float *gimg = a.img + (size_t)g * NB_IMG_COL128 * BS;
  if (tid == 0) *scount = 0;
  if (tid < 4 * BS) smask[tid] = 0u;
  // this thread's rays tid + i NT whose sums are weak in an image (bit k * R + i)
  constexpr int R = 4096 / NT;
  static_assert(R * BS <= 64, "a bit for each ray and image");
  unsigned long long cand = 0ull;
  bool flagged = false;
#pragma unroll
  for (int k = 0; k < BS; k++) {
    const float clip = sthr[k] * CLIP_QUANTA, all = sweak[k] ? sthr[k] * WEAK_QUANTA : 0.f;
    flagged |= sweak[k] != 0;
#pragma unroll
    for (int i = 0; i < R; i++) {
      const int ray = tid + i * NT;
      const float f = ray < 2 * a.nslots ? fabsf(vals[ray * BS + k]) : __int_as_float(0x7f800000);
      if (f < all || (f < clip && f > 0.f)) cand |= 1ull << (k * R + i);
    }
  }
  if (MODE == MODE_OSEM) {
    // where the randoms outweigh the error, or nothing was counted, the ratio does not need it
    float rs[R];
    int o[R];
    unsigned long long any = cand;
#pragma unroll
    for (int k = 1; k < BS; k++) any |= cand >> (k * R);
#pragma unroll
    for (int i = 0; i < R; i++) {
      const int ray = tid + i * NT;
      const nb_slot *S = a.slots + (ray >> 1);
      const int16_t *out = a.span == 11 ? &S->o11A : &S->o1A;
      o[i] = any >> i & 1u ? __ldg(out + (ray & 1)) : -1;
    }
#pragma unroll
    for (int i = 0; i < R; i++) rs[i] = o[i] >= 0 ? __ldg(a.rs + (size_t)lor * a.nout + o[i]) : 0.f;
#pragma unroll
    for (int k = 0; k < BS; k++) {
      const int rep = g * BS + k;
      const float q = sthr[k], scale = rep < a.nrep ? a.rscale[rep] : 0.f;
      const uint16_t *y = a.psng + ((size_t)(rep < a.nrep ? rep : 0) * a.naw + lor) * a.nout;
#pragma unroll
      for (int i = 0; i < R; i++)
        if (cand >> (k * R + i) & 1u) {
          const bool skip = o[i] < 0 || rep >= a.nrep || (q < __int_as_float(0x7f800000) &&
                            (scale * rs[i] >= q * WEAK_QUANTA || __ldg(y + o[i]) == 0));
          if (skip) cand &= ~(1ull << (k * R + i));
        }
    }
  }
  if (!__syncthreads_or(cand != 0ull)) return false;
  if (flagged) {
    const int e = tid % (128 * BS), q = e / BS, k = e % BS;
    const int z = natural ? q : (q < 64 ? 2 * q : 2 * (q - 64) + 1);
    const float lim = sthr[k] * WEAK_VALUE;
    bool hit = false;
    if (z < NB_IMZ)
#pragma unroll 8
      for (int s = tid / (128 * BS); s < n; s += NT / (128 * BS)) {
        const float v = __ldg(gimg + (size_t)scol[s] * stride + e);
        // (without a scale every value counts, NaN too)
        hit |= v != 0.f && (fabsf(v) < lim || lim == __int_as_float(0x7f800000));
      }
    if (hit) atomicOr(&smask[4 * k + (z & 1) * 2 + (z >> 6)], 1u << (z >> 1 & 31));
    __syncthreads();
  }
  const int last = n > 0 ? ((n - 1) >> 3) * 64 : 0;
#pragma unroll
  for (int i = 0; i < R; i++) {
    const int ray = tid + i * NT;
    bool weak = false;
#pragma unroll
    for (int k = 0; k < BS; k++)
      if (cand >> (k * R + i) & 1u) {
        const float f = fabsf(vals[ray * BS + k]);
        if (f > 0.f && f < sthr[k] * CLIP_QUANTA) {
          weak = true;
        } else {
          // the ray's planes, one more either side (its start plane may round away)
          const uint32_t zz = a.slots[ray >> 1].zzd;
          const int d = (int)(zz >> 16), m1 = rec[NB_REC_M + d] - 1, cnt = rec[NB_REC_KEND + last + d];
          const int z = ray & 1 ? (int)(zz >> 8 & 255u) - m1 : (int)(zz & 255u) + m1;
          weak |= mask_meets(smask + 4 * k, max(0, z - (ray & 1 ? cnt : 0) - 1),
                             min(127, z + (ray & 1 ? 0 : cnt) + 1));
        }
      }
    if (weak) list[atomicAdd(scount, 1)] = (uint16_t)ray;
  }
  __syncthreads();
  const int count = *scount;
  if (count == 0) return false;
  if (count <= NT / 8) {
    static_assert(NT / 8 * (NB_STEP_STRIDE / 8) * BS * 4 <= L::region - L::col_off, "block sums fit");
    walk_few<BS, NT>(gimg, stride, natural, scol, sst, n, h, a.slots, list, count, vals, cols);
    __syncthreads();
    return true;
  }
  for (int b0 = 0; b0 < count; b0 += NT) {
    const bool live = b0 + tid < count;
    const int ray = list[live ? b0 + tid : b0];
    nb_axial A;
    slot_axial(a.slots, ray, h, A);
    // offset of the ray's plane in a column (plane 127 reads as zero) and its change at the next
    // crossing; in the col128 order every second crossing turns between the even and odd halves
    int zo = (natural ? A.w : nb_zi(A.w)) * BS;
    int dz = natural ? A.dir : (A.dir > 0 ? ((A.w & 1) ? -63 : 64) : ((A.w & 1) ? -64 : 63)) * BS;
    const int dsum = natural ? 2 * A.dir : A.dir * BS;
    float tp = h.x, tzc = A.tzc, acc[BS], sum[BS];   // of a block of 8 steps; of the blocks
#pragma unroll
    for (int k = 0; k < BS; k++) sum[k] = 0.f;
    for (int s0 = 0; s0 < n; s0 += L::ncol) {
      const int m = min(L::ncol, n - s0);
      __syncthreads();                        // the columns before have been walked
      for (int x = tid; x < m * 128; x += NT)
        if (!natural || (x & 127) < NB_IMZ)
          nb_cp_async<4 * BS>(cols + x * BS, gimg + (size_t)scol[s0 + (x >> 7)] * stride + (x & 127) * BS);
        else
          cols[x] = 0.f;
      nb_cp_async_wait();
      __syncthreads();
      if (!live) continue;
      const float *c = cols + zo;
      auto step = [&](int u, float tn) {
        float v[BS];
        ldv<BS>(c + u * 128 * BS, v);
        const float w = __fsub_rn(fminf(tn, tzc), tp);
#pragma unroll
        for (int k = 0; k < BS; k++) acc[k] = fmaf(w, v[k], acc[k]);
        if (tn > tzc) {
          c += dz;
          dz = dsum - dz;
          ldv<BS>(c + u * 128 * BS, v);
          const float w1 = __fsub_rn(tn, tzc);
#pragma unroll
          for (int k = 0; k < BS; k++) acc[k] = fmaf(w1, v[k], acc[k]);
          tzc = __fadd_rn(tzc, A.dtz);
        }
        tp = tn;
      };
      int i = 0;
      for (; i + 8 <= m; i += 8) {
        float t[8];
        ldv<4>(sst + s0 + i, t);
        ldv<4>(sst + s0 + i + 4, t + 4);
#pragma unroll
        for (int k = 0; k < BS; k++) acc[k] = 0.f;
#pragma unroll
        for (int u = 0; u < 8; u++) step(u, t[u]);
#pragma unroll
        for (int k = 0; k < BS; k++) sum[k] += acc[k];
        c += 8 * 128 * BS;
      }
      if (i < m) {
#pragma unroll
        for (int k = 0; k < BS; k++) acc[k] = 0.f;
        for (; i < m; i++) {
          step(0, sst[s0 + i]);
          c += 128 * BS;
        }
#pragma unroll
        for (int k = 0; k < BS; k++) sum[k] += acc[k];
      }
      zo = (int)(c - cols) - m * 128 * BS;
    }
    if (live)
#pragma unroll
      for (int k = 0; k < BS; k++) vals[ray * BS + k] = sum[k];
  }
  __syncthreads();
  return true;
}

// Back projection of a LOR's values (vals, [4096][BS]) for the images of `which`: step by step in
// float32, straight into the image.  For values without a fixed-point scale, which reach the
// voxels of their rays and no others.  All threads.
template <int BS, int NT, class L>
static __device__ __forceinline__ void spread_rays(const WalkArgs &a, unsigned char *smem, int par,
                                                int g, int n, const float4 h, unsigned which) {
  const int32_t *scol = reinterpret_cast<const int32_t *>(
      smem + L::cs_off + (size_t)par * 8 * NB_STEP_STRIDE);
  const float *sst = reinterpret_cast<const float *>(scol) + NB_STEP_STRIDE;
  const float *vals = reinterpret_cast<const float *>(smem);
  float *gb = a.bimg + (size_t)g * NB_IMG_COL128 * BS;
  for (int ray = threadIdx.x; ray < 2 * a.nslots; ray += NT) {
    nb_axial A;
    slot_axial(a.slots, ray, h, A);
    for (int k = 0; k < BS; k++) {
      const float v = vals[ray * BS + k];
      if (!(which >> k & 1u) || v == 0.f) continue;
      int z = A.w;
      float tp = h.x, tzc = A.tzc;
      auto add = [&](int s, float w) {        // plane 127 is padding
        if (w != 0.f && z < NB_IMZ)
          atomicAdd(gb + ((size_t)scol[s] * NB_COLW + nb_zi(z)) * BS + k, w * v);
      };
      for (int s = 0; s < n; s++) {
        const float tn = sst[s];
        add(s, __fsub_rn(fminf(tn, tzc), tp));
        if (tn > tzc) {
          z += A.dir;
          add(s, __fsub_rn(tn, tzc));
          tzc = __fadd_rn(tzc, A.dtz);
        }
        tp = tn;
      }
    }
  }
}

template <int BS, int CH, int NT, int MODE, int MINB>
__global__ void __launch_bounds__(NT, MINB) k_walk(const __grid_constant__ WalkArgs a) {
  constexpr int NSEG = NT / 64;               // step segments of a chunk, one per 64 threads
  constexpr int SEGL = CH / NSEG;
  constexpr int SPT = (NB_NSLOT + NT - 1) / NT;          // slots (ray pairs) per thread
  constexpr int W = NT / 32;
  constexpr int UNIT = BS == 1 ? 8 : 16;      // bytes per plane of a table row
  constexpr int LOGR = BS == 1 ? 10 : (BS == 2 ? 11 : 12);   // table row bytes
  constexpr int LOGG = LOGR - 1;                             // accumulator row bytes
  static_assert(CH % 8 == 0 && CH % NSEG == 0 && SEGL >= 1, "chunk shape");
  static_assert(NSEG * BS % 4 == 0, "the bounds are read 16 bytes at a time");
  using L = WSmem<BS, CH, NSEG>;
  extern __shared__ __align__(1024) unsigned char smem[];
  unsigned char *tab = smem;
  int *gacc = reinterpret_cast<int *>(smem);
  float *stage = reinterpret_cast<float *>(smem + L::stg_off);
  float *vals = reinterpret_cast<float *>(smem);                     // [4096][BS]
  int *sseg = reinterpret_cast<int *>(smem + L::seg_off);
  int *soc = reinterpret_cast<int *>(smem + L::oc_off);              // prefixes of voxel 63
  int *srun = reinterpret_cast<int *>(smem + L::run_off);
  unsigned char *rec = smem + L::rec_off;
  float *sobl = reinterpret_cast<float *>(smem + L::obl_off);        // oblique length factors
  unsigned char *misc = smem + L::misc_off;
  uint64_t *bar = reinterpret_cast<uint64_t *>(misc);
  uint64_t *bar2 = reinterpret_cast<uint64_t *>(misc + 8);
  void *clc = misc + 16;                                             // launch control's answer
  int *sflag = reinterpret_cast<int *>(misc + 32);
  int *snext = reinterpret_cast<int *>(misc + 36);
  unsigned *smax = reinterpret_cast<unsigned *>(smem + L::max_off);  // forward bounds
  unsigned *smaxb = reinterpret_cast<unsigned *>(misc + 64);         // [2][BS] backward
  float *sthr = reinterpret_cast<float *>(misc + 96);                // [BS] sum of the quanta
  int *sweak = reinterpret_cast<int *>(misc + 112);                  // [BS] weak values were met
  unsigned *smin = reinterpret_cast<unsigned *>(misc + 128);         // [3][BS] least |value|

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int s = tid & 63;                     // scan: this thread's planes 2 s and 2 s + 1
  const int seg = tid >> 6;                   // ... in this segment
  const uint32_t tab_u = nb_smem_u32(tab), rec_u = nb_smem_u32(rec);
  const bool span11 = a.span == 11;

  if (tid == 0) {
    nb_mbar_init(bar, 1);
    nb_mbar_init(bar2, 1);
    *sflag = 0;
    for (int k = 0; k < 3 * NSEG * BS; k++) smax[k] = 0u;
    for (int k = 0; k < 3 * BS; k++) smin[k] = ~0u;
    for (int k = 0; k < 2 * BS; k++) smaxb[k] = 0u;
    nb_fence_mbar_init();
  }
  if (MODE == MODE_BWD)
    for (int i = tid; i < (CH + 1) * 128 * BS; i += NT) gacc[i] = 0;
  __syncthreads();

  // one thread: the record, columns and exit parameters of job q into shared memory
  auto issue = [&](int q, int buf) {
    const int p = q / a.ngroups;
    int lor = a.subs ? a.subs[p] : p;
    if (lor < 0 || lor >= a.naw) {
      nb_set_error(a.err, NB_DEVERR_BAD_LOR);
      lor = 0;
    }
    const int n = __float_as_int(a.hdr[lor].w);
    const uint32_t r0 = a.rec_off[lor], rb = (a.rec_off[lor + 1] - r0) * 16u;
    const uint32_t cb = max(16u, (uint32_t)((n * 4 + 15) & ~15));
    unsigned char *cs = smem + L::cs_off + (size_t)buf * 8 * NB_STEP_STRIDE;
    nb_mbar_arrive_expect_tx(bar, rb + 2 * cb);
    nb_bulk_g2s(rec, a.rec + (size_t)r0 * 16, rb, bar);
    nb_bulk_g2s(cs, a.scol + (size_t)lor * NB_STEP_STRIDE, cb, bar);
    nb_bulk_g2s(cs + 4 * NB_STEP_STRIDE, a.st + (size_t)lor * NB_STEP_STRIDE, cb, bar);
  };
  // The grid has one block per job (LOR, image group); a block that has finished takes over
  // a job whose block has not started, so that long and short LORs even out over the SMs and
  // the next LOR's copies are in flight while this one ends.
  auto next_job = [&](int job) {
    int q = -1;
    if (nb_mbar_wait(bar2, (uint32_t)(job & 1), WAIT_POLLS)) {
      q = nb_clc_answer(clc);
      nb_fence_proxy_async_smem();   // the answer is read before the next request rewrites it
    } else {
      nb_set_error(a.err, NB_DEVERR_MBAR_TIMEOUT);
    }
    *snext = q;
    if (q >= 0) {
      issue(q, (job + 1) & 1);
      if (MODE != MODE_FWD) {                // the next job's rows, into L2 (two images: 1%)
        const int p = q / a.ngroups, g = q - p * a.ngroups;
        int lor = a.subs ? a.subs[p] : p;
        lor = lor < 0 || lor >= a.naw ? 0 : lor;
        auto row = [](const void *x, size_t bytes) {
          const uintptr_t a0 = ((uintptr_t)x + 15) & ~(uintptr_t)15, a1 = ((uintptr_t)x + bytes) & ~(uintptr_t)15;
          if (a1 > a0) nb_bulk_prefetch_l2((const void *)a0, (uint32_t)(a1 - a0));
        };
        for (int k = 0; k < BS; k++) {
          const int rep = g * BS + k;
          if (rep >= a.nrep) break;
          if (MODE == MODE_BWD)
            row(a.sino_in + ((size_t)rep * a.nprj + (a.in_by_lor ? lor : p)) * a.nout, 4 * (size_t)a.nout);
          else
            row(a.psng + ((size_t)rep * a.naw + lor) * a.nout, 2 * (size_t)a.nout);
        }
        if (MODE == MODE_OSEM) row(a.rs + (size_t)lor * a.nout, 4 * (size_t)a.nout);
      }
    }
  };
  if (tid == 0) issue(blockIdx.x, 0);

  int mrot = 0, q = blockIdx.x;
  for (int job = 0; q >= 0; job++) {
    const int p = q / a.ngroups, g = q - p * a.ngroups;
    const int lor0 = a.subs ? a.subs[p] : p;
    const bool badlor = lor0 < 0 || lor0 >= a.naw;
    const int lor = badlor ? 0 : lor0;
    const float4 h = a.hdr[lor];
    const int n = badlor ? 0 : __float_as_int(h.w);
    const int nch = (n + CH - 1) / CH;
    const int32_t *scol = reinterpret_cast<const int32_t *>(
        smem + L::cs_off + (size_t)(job & 1) * 8 * NB_STEP_STRIDE);
    const float *sst = reinterpret_cast<const float *>(scol) + NB_STEP_STRIDE;
    const float *gimg = MODE == MODE_BWD ? nullptr : a.img + (size_t)g * NB_IMG_COL128 * BS;

    if (!nb_mbar_wait(bar, (uint32_t)(job & 1), WAIT_POLLS)) atomicExch(sflag, 1);
    if (MODE != MODE_FWD && warp == 0) nb_bulk_wait_read<0>();   // staging region reusable
    __syncthreads();
    if (*sflag) break;
    if (tid == 0) nb_clc_request(clc, bar2);
    if (MODE != MODE_BWD && tid == 0)         // (this thread alone writes them)
      for (int k = 0; k < BS; k++) sthr[k] = 0.f, sweak[k] = 0;

    auto slot_of = [&](int j) { return ((j & 1) ? (j + 1) * W - 1 - warp : j * W + warp) * 32 + lane; };
    // lengths of this thread's steps in the chunk at s0 (0 past the LOR's end, where the reads
    // find other data of the block)
    auto step_lengths = [&](int s0, float *lt) {
      float t[SEGL];
      const int f0 = s0 + seg * SEGL;
      if (SEGL % 4 == 0) {
#pragma unroll
        for (int j = 0; j < SEGL; j += 4) ldv<4>(sst + f0 + j, t + j);
      } else {
#pragma unroll
        for (int j = 0; j < SEGL; j++) t[j] = sst[f0 + j];
      }
      float tp = f0 ? sst[f0 - 1] : h.x;
#pragma unroll
      for (int j = 0; j < SEGL; j++) {
        lt[j] = f0 + j < n ? __fsub_rn(t[j], tp) : 0.f;
        tp = t[j];
      }
    };

    // this thread's slots: start planes of the two rays (8 bits each) and crossing schedule (the
    // ring difference, but for the few pairs listed in the record)
    uint32_t zzd[SPT];
    const int nirr = *reinterpret_cast<const uint16_t *>(rec + NB_REC_META);
#pragma unroll
    for (int j = 0; j < SPT; j++) {
      const int sl = slot_of(j);
      zzd[j] = 0u;
      if (sl >= a.nslots) continue;
      const uint32_t zz = __ldg(&a.slots[sl].zzd);
      uint32_t id = zz >> 16, off = 0u;
      for (int x = 0; x < nirr; x++) {
        const char4 e = reinterpret_cast<const char4 *>(rec + NB_REC_IRR)[x];
        if (e.x == (int)(zz >> 16) && 2 * (int)e.y == (int)(zz & 255u)) {
          if (e.z == 2)
            id = (uint32_t)e.w;
          else
            off += (uint32_t)(e.z ? 256 * (int)e.w : (int)e.w);
        }
      }
      // the upward ray starts m - 1 planes above its ring's, the downward one as many below
      zzd[j] = (zz & 0xffffu) - (uint32_t)(rec[NB_REC_M + id] - 1) * 255u + off + (id << 16);
    }
    if (tid < 64)
      sobl[tid] = oblique_s(tid <= NB_MAXRD ? tid : rec[NB_REC_META + 2 + tid - NB_MAXRD - 1], h.y);
    if (MODE == MODE_BWD) __syncthreads();           // (the forward pass has later barriers)

    float FA[SPT][BS], FB[SPT][BS];           // forward: line integrals
#pragma unroll
    for (int j = 0; j < SPT; j++)
#pragma unroll
      for (int k = 0; k < BS; k++) FA[j][k] = FB[j][k] = 0.f;

    // ------------------------------------------------------------------ forward
    if (MODE != MODE_BWD) {
      float E[SEGL][BS], O[SEGL][BS];         // this thread's values: planes 2 s, 2 s + 1
      const bool natural = MODE == MODE_FWD && BS == 1 && a.natural != 0;
      auto load = [&](int c) {
        int col[SEGL];
        const int f0 = c * CH + seg * SEGL;
        if (SEGL % 4 == 0) {
#pragma unroll
          for (int j = 0; j < SEGL; j += 4) ldi<4>(scol + f0 + j, col + j);
        } else {
#pragma unroll
          for (int j = 0; j < SEGL; j++) col[j] = scol[f0 + j];
        }
#pragma unroll
        for (int j = 0; j < SEGL; j++) {
          if (f0 + j < n) {
            const float *x = gimg + (size_t)col[j] * (natural ? NB_IMZ : NB_COLW * BS) +
                             (natural ? 2 * s : s * BS);
            ldg_v<BS>(x, E[j]);
            if (natural && s == 63)
              O[j][0] = 0.f;
            else
              ldg_v<BS>(x + (natural ? 1 : 64 * BS), O[j]);
          } else {
#pragma unroll
            for (int v = 0; v < BS; v++) E[j][v] = O[j][v] = 0.f;
          }
        }
      };
      for (int c = 0; c < nch; c++) {
        const int s0 = c * CH, s1 = min(n, s0 + CH);
        // (holding the next chunk's values through the walk instead hid their latency but
        // spilled: 1604 against 1487 us for one image's fused subset, 1471 against 1267 for two)
        load(c);
        // bound of the chunk's integrals per image: over its segments, the largest integral
        // of |value| of any plane
        float lt[SEGL];
        {
          step_lengths(s0, lt);
          float m[BS];
#pragma unroll
          for (int v = 0; v < BS; v++) m[v] = 0.f;
#pragma unroll
          for (int v = 0; v < BS; v++) {
            float me = 0.f, mo = 0.f;
#pragma unroll
            for (int j = 0; j < SEGL; j++) {
              me = fmaf(lt[j], fabsf(E[j][v]), me);
              mo = fmaf(lt[j], fabsf(O[j][v]), mo);
            }
            const unsigned u = __reduce_max_sync(0xffffffffu, max(__float_as_uint(me), __float_as_uint(mo)));
            if (u == 0u) continue;            // (the whole warp)
            unsigned lo = ~0u;                // least non-zero |value|, as 2 * bits - 1
#pragma unroll
            for (int j = 0; j < SEGL; j++)
              lo = min(lo, min(2u * __float_as_uint(E[j][v]) - 1u, 2u * __float_as_uint(O[j][v]) - 1u));
            lo = __reduce_min_sync(0xffffffffu, lo);
            if (lane == 0) {
              atomicMax(&smax[(mrot * NSEG + seg) * BS + v], u);
              atomicMin(&smin[mrot * BS + v], lo);
            }
          }
        }
        __syncthreads();
        unsigned any = 0u;
        float scale[BS], inv[BS], bnd[NSEG * BS];
#pragma unroll
        for (int x = 0; x < NSEG * BS; x += 4)
          ldv<4>(reinterpret_cast<const float *>(smax) + mrot * NSEG * BS + x, bnd + x);
#pragma unroll
        for (int k = 0; k < BS; k++) {
          float bound = 0.f;
#pragma unroll
          for (int x = 0; x < NSEG; x++) bound += bnd[x * BS + k];
          const unsigned bb = __float_as_uint(bound);
          any |= bb;
          // bound < 2^e: scale 2^(29 - e), as far as float32 has it.  A bound that is not finite or
          // above 2^100 has none: the image's rays are all walked again
          const int x = min(155 - (int)(bb >> 23), 126);
          const bool none = bb >= 0x71800000u;
          scale[k] = bb && !none ? __uint_as_float((uint32_t)(127 + x) << 23) : 0.f;
          inv[k] = bb && !none ? __uint_as_float((uint32_t)(127 - x) << 23) : 0.f;
          if (bb != 0u && tid == 0) {
            sthr[k] += none ? __int_as_float(0x7f800000) : inv[k];
            if (none || smin[mrot * BS + k] < 2u * __float_as_uint(inv[k] * WEAK_VALUE) - 1u) sweak[k] = 1;
          }
        }
        // cleared two chunks before its next use: its last readers are one barrier back
        if (tid < NSEG * BS) smax[((mrot + 2) % 3) * NSEG * BS + tid] = 0u;
        if (tid < BS) smin[((mrot + 2) % 3) * BS + tid] = ~0u;
        mrot = (mrot + 1) % 3;
        if (any == 0u) continue;              // nothing but zeros
        {
          // fixed-point running integrals: within the segment, then the segments before it
          // (rounded with offsets spread over (-1/2, 1/2), so that the errors of equal values do
          // not add up; 0 stays 0)
          int cE[SEGL][BS], cO[SEGL][BS], tE[BS], tO[BS];
#pragma unroll
          for (int v = 0; v < BS; v++) tE[v] = tO[v] = 0;
#pragma unroll
          for (int j = 0; j < SEGL; j++) {
            const float off = (float)(2 * ((5 * j + 2) % 8) - 7) / 16.f;
#pragma unroll
            for (int v = 0; v < BS; v++) {
              const float w = lt[j] * scale[v];
              cE[j][v] = tE[v];
              cO[j][v] = tO[v];
              tE[v] += __float2int_rn(fmaf(E[j][v], w, off));
              tO[v] += __float2int_rn(fmaf(O[j][v], w, off));
            }
            if (s == 31) sti<BS>(soc + (seg * (SEGL + 1) + j) * BS, cO[j]);
          }
          if (s == 31) sti<BS>(soc + (seg * (SEGL + 1) + SEGL) * BS, tO);
          sti<BS>(sseg + (seg * 128 + s) * BS, tE);
          sti<BS>(sseg + (seg * 128 + 64 + s) * BS, tO);
          __syncthreads();
          int bE[BS], bO[BS];
#pragma unroll
          for (int v = 0; v < BS; v++) bE[v] = bO[v] = 0;
          for (int x = 0; x < seg; x++) {
            int u[BS], w[BS];
            ldi<BS>(sseg + (x * 128 + s) * BS, u);
            ldi<BS>(sseg + (x * 128 + 64 + s) * BS, w);
#pragma unroll
            for (int v = 0; v < BS; v++) bE[v] += u[v], bO[v] += w[v];
          }
          // the thread of plane 64 gets plane 63's prefixes through shared memory (its neighbour
          // is another warp's); the thread of plane 0 has no plane below and its D[0] no reader
          const bool fix = s == 32;
          int bP[BS];
#pragma unroll
          for (int v = 0; v < BS; v++) bP[v] = 0;
          if (fix)
            for (int x = 0; x < seg; x++) {
              int u[BS];
              ldi<BS>(sseg + (x * 128 + 64 + 31) * BS, u);
#pragma unroll
              for (int v = 0; v < BS; v++) bP[v] += u[v];
            }
          if (seg == NSEG - 1) {              // the chunk's whole integral per plane
            int u[BS], w[BS];
#pragma unroll
            for (int v = 0; v < BS; v++) u[v] = tE[v] + bE[v], w[v] = tO[v] + bO[v];
            sti<BS>(srun + s * BS, u);
            sti<BS>(srun + (64 + s) * BS, w);
          }
          // D at the start of each step and its change over the step
          int De[BS], Do[BS];
#pragma unroll
          for (int j = SEGL; j >= 0; j--) {
            int ne[BS], no[BS];               // D at the end of step j
#pragma unroll
            for (int v = 0; v < BS; v++) {
              ne[v] = De[v];
              no[v] = Do[v];
              const int ce = (j < SEGL ? cE[j < SEGL ? j : 0][v] : tE[v]) + bE[v];
              const int co = (j < SEGL ? cO[j < SEGL ? j : 0][v] : tO[v]) + bO[v];
              int cp = __shfl_up_sync(0xffffffffu, co, 1);      // plane 2 s - 1
              if (fix) cp = bP[v] + soc[(seg * (SEGL + 1) + j) * BS + v];
              De[v] = cp - ce;
              Do[v] = ce - co;
              ne[v] -= De[v];
              no[v] -= Do[v];
            }
            if (j == SEGL) continue;
            unsigned char *r = tab + ((size_t)(seg * SEGL + j) << LOGR) + s * UNIT;
            if (BS == 1) {
              *reinterpret_cast<int2 *>(r) = make_int2(De[0], ne[0]);
              *reinterpret_cast<int2 *>(r + 64 * UNIT) = make_int2(Do[0], no[0]);
            } else if (BS == 2) {
              *reinterpret_cast<int4 *>(r) = make_int4(De[0], De[BS - 1], ne[0], ne[BS - 1]);
              *reinterpret_cast<int4 *>(r + 64 * UNIT) = make_int4(Do[0], Do[BS - 1], no[0], no[BS - 1]);
            } else {
              sti<BS>(reinterpret_cast<int *>(r), De);
              sti<BS>(reinterpret_cast<int *>(r + 64 * UNIT), Do);
              sti<BS>(reinterpret_cast<int *>(r + 2048), ne);
              sti<BS>(reinterpret_cast<int *>(r + 2048 + 64 * UNIT), no);
            }
          }
          __syncthreads();
        }

        const unsigned char *kend = rec + NB_REC_KEND;
        const int krow0 = c * (CH / 8) - 1, krow1 = (s1 - 1) >> 3;
#pragma unroll
        for (int j = 0; j < SPT; j++) {
          const int zz = (int)zzd[j], d = zz >> 16;
          const int ka = c ? kend[krow0 * 64 + d] : 0;
          int cnt = kend[krow1 * 64 + d] - ka;
          const int e0 = reinterpret_cast<const uint16_t *>(rec + NB_REC_OFF)[d] + ka;
          const int zA = (zz & 255) + ka, zB = ((zz >> 8) & 255) - ka;
          const int endA = zA + cnt, endB = zB - cnt;
          uint32_t ep = rec_u + NB_REC_ENT + e0 * 8;
          // cursors of the next crossing and the one after (their plane offsets in a row);
          // two crossings on, both have moved by one unit
          const uint32_t base = tab_u - ((uint32_t)s0 << LOGR);
          uint32_t cA0 = base + plane_off(zA + 1, UNIT), cB0 = base + plane_off(zB, UNIT);
          uint32_t cA1 = cA0 + 64 * UNIT - ((zA + 1) & 1) * (127 * UNIT);
          uint32_t cB1 = cB0 + 63 * UNIT - (zB & 1) * (127 * UNIT);
          // sums of D + dD * fraction in 2^-QBITS quanta, 64 bits: a ray that changes planes can
          // collect more than any plane holds, up to SEGL times 2^29.  Two crossings' D fit 32
          // (the plane between them cancels but for what the ray collects in it: 3 x 2^29)
          long long xA[BS], xB[BS];
          int dA[BS], dB[BS];
#pragma unroll
          for (int k = 0; k < BS; k++) xA[k] = xB[k] = 0;
          auto cross = [&](int f, uint32_t rA, uint32_t rB) {
            int X[BS];
            lds_tab<BS>(rA, dA, X);
#pragma unroll
            for (int k = 0; k < BS; k++) xA[k] += (long long)X[k] * f;
            lds_tab<BS>(rB, dB, X);
#pragma unroll
            for (int k = 0; k < BS; k++) xB[k] += (long long)X[k] * f;
          };
          for (; cnt >= 2; cnt -= 2) {
            int i0, i1, f0, f1, eA[BS], eB[BS];
            lds_ent(ep, i0, f0);
            lds_ent(ep + 8, i1, f1);
            ep += 16;
            cross(f0, cA0 + (i0 << LOGR), cB0 + (i0 << LOGR));
#pragma unroll
            for (int k = 0; k < BS; k++) eA[k] = dA[k], eB[k] = dB[k];
            cross(f1, cA1 + (i1 << LOGR), cB1 + (i1 << LOGR));
#pragma unroll
            for (int k = 0; k < BS; k++) {
              xA[k] += (long long)(eA[k] + dA[k]) * (1 << QBITS);
              xB[k] += (long long)(eB[k] + dB[k]) * (1 << QBITS);
            }
            cA0 += UNIT;
            cA1 += UNIT;
            cB0 -= UNIT;
            cB1 -= UNIT;
          }
          if (cnt) {
            int i0, f0;
            lds_ent(ep, i0, f0);
            cross(f0, cA0 + (i0 << LOGR), cB0 + (i0 << LOGR));
#pragma unroll
            for (int k = 0; k < BS; k++) {
              xA[k] += (long long)dA[k] * (1 << QBITS);
              xB[k] += (long long)dB[k] * (1 << QBITS);
            }
          }
          // the down-going ray leaves C[P] for C[P-1]: its differences count negative
          int u[BS], w[BS];
          ldi<BS>(srun + nb_zi(endA) * BS, u);
          ldi<BS>(srun + nb_zi(endB) * BS, w);
#pragma unroll
          for (int k = 0; k < BS; k++) {
            FA[j][k] = fmaf(quanta(u[k], xA[k]), inv[k], FA[j][k]);
            FB[j][k] = fmaf(quanta(w[k], -xB[k]), inv[k], FB[j][k]);
          }
        }
      }
      // rays whose sums are too few quanta to be good to float32's precision are walked again
      bool weak = false;
#pragma unroll
      for (int k = 0; k < BS; k++) {
        const float clip = sthr[k] * CLIP_QUANTA, all = sweak[k] ? sthr[k] * WEAK_QUANTA : 0.f;
#pragma unroll
        for (int j = 0; j < SPT; j++) {
          const float fA = fabsf(FA[j][k]), fB = fabsf(FB[j][k]);
          weak |= fA < all || (fA < clip && fA > 0.f) || fB < all || (fB < clip && fB > 0.f);
        }
      }
      bool again = __syncthreads_or(weak);    // (the walk is done: the table region is free)
      if (MODE == MODE_OSEM && again) again = __syncthreads_or(bins_matter<BS, NT>(a, sthr, g, lor));
      if (again) {
#pragma unroll
        for (int j = 0; j < SPT; j++) {
          const int sl = slot_of(j);
          if (sl >= a.nslots) continue;
#pragma unroll
          for (int k = 0; k < BS; k++) {
            vals[2 * sl * BS + k] = FA[j][k];
            vals[(2 * sl + 1) * BS + k] = FB[j][k];
          }
        }
        __syncthreads();
        if (walk_weak<BS, NT, MODE, L>(a, smem, job & 1, g, lor, n, h)) {
#pragma unroll
          for (int j = 0; j < SPT; j++) {
            const int sl = slot_of(j);
            if (sl >= a.nslots) continue;
            ldv<BS>(vals + 2 * sl * BS, FA[j]);
            ldv<BS>(vals + (2 * sl + 1) * BS, FB[j]);
          }
          __syncthreads();
        }
      }
      if (MODE == MODE_FWD && tid == 0) next_job(job);   // the record is free

      // ratio of a bin (recon.cu:459-470): y / (Ax + rscale (r+s)/(an)), 0 where |.| < 1e-6
      auto ratio = [&](float v, int o, int k) {
        const int rep = g * BS + k;
        if (rep >= a.nrep) return 0.f;
        const size_t gi = (size_t)lor * a.nout + o;
        const float e = v + a.rscale[rep] * a.rs[gi];
        const float y = (float)a.psng[(size_t)rep * a.naw * a.nout + gi];
        return (e > -0.000001f && e < 0.000001f) ? 0.f : __fdiv_rn(y, e);
      };
#pragma unroll
      for (int j = 0; j < SPT; j++) {
        const int sl = slot_of(j);
        if (sl >= a.nslots) continue;
        const nb_slot *S = a.slots + sl;
        const float so = sobl[zzd[j] >> 16];
        int oA = 0, oB = 0;
        if (!span11) oA = S->o1A, oB = S->o1B;
#pragma unroll
        for (int k = 0; k < BS; k++) {
          float vA = FA[j][k] * so, vB = FB[j][k] * so;
          if (MODE == MODE_FWD && a.att == 1) {
            vA = expf(-vA);
            vB = expf(-vB);
            if (span11) {
              vA = vA / (float)S->nosA;
              vB = vB / (float)S->nosB;
            }
          }
          if (span11) {
            vals[(2 * sl) * BS + k] = vA;
            vals[(2 * sl + 1) * BS + k] = vB;
          } else if (MODE == MODE_FWD) {
            const int rep = g * BS + k;
            if (rep < a.nrep) {
              float *row = a.sino + ((size_t)rep * a.nprj + p) * a.nout;
              if (oA >= 0) row[oA] = vA;
              if (oB >= 0) row[oB] = vB;
            }
          } else {
            FA[j][k] = oA >= 0 ? ratio(vA, oA, k) : 0.f;
            FB[j][k] = oB >= 0 ? ratio(vB, oB, k) : 0.f;
          }
        }
      }
      if (span11) {
        __syncthreads();
        for (int x = tid; x < a.nout * BS; x += NT) {
          const int o = x / BS, k = x - o * BS;
          float v = 0.f;
          const int4 l4 = __ldg(reinterpret_cast<const int4 *>(a.bin11 + o * 8));
          const int16_t *lst = reinterpret_cast<const int16_t *>(&l4);
#pragma unroll
          for (int r = 0; r < 8; r++)
            if (lst[r] >= 0) v += vals[lst[r] * BS + k];
          if (MODE == MODE_FWD) {
            const int rep = g * BS + k;
            if (rep < a.nrep) a.sino[((size_t)rep * a.nprj + p) * a.nout + o] = v;
          } else {
            // back to the bin's rays (a ray is in one bin; its integral is not read again)
            v = ratio(v, o, k);
#pragma unroll
            for (int r = 0; r < 8; r++)
              if (lst[r] >= 0) vals[lst[r] * BS + k] = v;
          }
        }
        if (MODE == MODE_OSEM) __syncthreads();
      }
    }

    // ------------------------------------------------------------------ backward
    if (MODE != MODE_FWD) {
      // values to spread and their fixed-point scale, per image (images of one group can
      // differ in count level by orders of magnitude)
      unsigned mm[BS];                        // largest |value|, as bits (NaN above infinity)
#pragma unroll
      for (int k = 0; k < BS; k++) mm[k] = 0u;
#pragma unroll
      for (int j = 0; j < SPT; j++) {
        const int sl = slot_of(j);
        if (sl >= a.nslots) {                 // lanes without a pair have walked plane 0
#pragma unroll
          for (int k = 0; k < BS; k++) FA[j][k] = FB[j][k] = 0.f;
          continue;
        }
        const short2 o2 = __ldg(reinterpret_cast<const short2 *>(span11 ? &a.slots[sl].o11A : &a.slots[sl].o1A));
        const float so = sobl[zzd[j] >> 16];
        const int oA = o2.x, oB = o2.y;
#pragma unroll
        for (int k = 0; k < BS; k++) {
          if (MODE == MODE_BWD) {
            const int rep = g * BS + k;
            const float *row =
                a.sino_in + ((size_t)rep * a.nprj + (a.in_by_lor ? lor : p)) * a.nout;
            FA[j][k] = oA >= 0 && rep < a.nrep ? row[oA] : 0.f;
            FB[j][k] = oB >= 0 && rep < a.nrep ? row[oB] : 0.f;
          } else if (span11) {
            FA[j][k] = oA >= 0 ? vals[(2 * sl) * BS + k] : 0.f;
            FB[j][k] = oB >= 0 ? vals[(2 * sl + 1) * BS + k] : 0.f;
          }
          FA[j][k] *= so;
          FB[j][k] *= so;
          mm[k] = max(mm[k], max(__float_as_uint(fabsf(FA[j][k])), __float_as_uint(fabsf(FB[j][k]))));
        }
      }
      const int par = job & 1;
#pragma unroll
      for (int k = 0; k < BS; k++) {
        const unsigned m = __reduce_max_sync(0xffffffffu, mm[k]);
        if (lane == 0 && m) atomicMax(&smaxb[par * BS + k], m);
      }
      for (int i = tid; i < 128 * BS; i += NT) srun[i] = 0;
      __syncthreads();
      if (MODE == MODE_OSEM)                  // (the ratios have been read; a barrier follows)
        for (int i = tid; i < (CH + 1) * 32 * BS; i += NT)
          reinterpret_cast<int4 *>(gacc)[i] = make_int4(0, 0, 0, 0);
      unsigned none = 0u;                     // images without a scale: a value is not finite
#pragma unroll
      for (int k = 0; k < BS; k++) none |= (smaxb[par * BS + k] >= 0x7f800000u ? 1u : 0u) << k;
      if (none) {
        // these images' rays one by one, through the accumulators' memory
        __syncthreads();
#pragma unroll
        for (int j = 0; j < SPT; j++) {
          const int sl = slot_of(j);
          if (sl >= a.nslots) continue;
#pragma unroll
          for (int k = 0; k < BS; k++) {
            vals[2 * sl * BS + k] = FA[j][k];
            vals[(2 * sl + 1) * BS + k] = FB[j][k];
          }
        }
        __syncthreads();
        spread_rays<BS, NT, L>(a, smem, job & 1, g, n, h, none);
        __syncthreads();
        for (int i = tid; i < (CH + 1) * 128 * BS; i += NT) gacc[i] = 0;
        __syncthreads();
      }
      float inv[BS];
      int VA[SPT][BS], VB_[SPT][BS];          // the rays' values, integers
      unsigned any = 0u;
#pragma unroll
      for (int k = 0; k < BS; k++) {
        const unsigned mb = smaxb[par * BS + k];
        float sc = 0.f;
        inv[k] = 0.f;
        if (mb != 0u && mb < 0x7f800000u) {
          const int e = max((int)(mb >> 23) - 126, -96);   // max < 2^e
          sc = __uint_as_float((uint32_t)(FXBITS - e + 127) << 23);
          inv[k] = __uint_as_float((uint32_t)(e - FXBITS + 127) << 23);
          any = 1u;
        }
#pragma unroll
        for (int j = 0; j < SPT; j++) {
          VA[j][k] = __float2int_rn(FA[j][k] * sc);
          VB_[j][k] = __float2int_rn(FB[j][k] * sc);
        }
      }
      if (tid < BS) smaxb[(par ^ 1) * BS + tid] = 0u;
      const int nchb = any ? nch : 0;         // 0: nothing to spread
      if (nchb == 0) {
        __syncthreads();
        if (tid == 0) next_job(job);
      }
      const uint32_t g_u = nb_smem_u32(gacc), run_u = nb_smem_u32(srun);
#pragma unroll
      for (int j = 0; j < SPT && nchb; j++) {
        const int zA = zzd[j] & 255, zB = (zzd[j] >> 8) & 255;
#pragma unroll
        for (int k = 0; k < BS; k++) {
          const int vA = VA[j][k], vB = VB_[j][k];
          if (vA) reds_add_s32(run_u + (nb_zi(zA) * BS + k) * 4, vA);
          if (vB) reds_add_s32(run_u + (nb_zi(zB) * BS + k) * 4, vB);
        }
      }
      if (MODE == MODE_OSEM) __syncthreads();
      float *gb = a.bimg + (size_t)g * NB_IMG_COL128 * BS;
      for (int c = 0; c < nchb; c++) {
        const int s0 = c * CH, s1 = min(n, s0 + CH);
        const unsigned char *kend = rec + NB_REC_KEND;
        const int krow0 = c * (CH / 8) - 1, krow1 = (s1 - 1) >> 3;
#pragma unroll
        for (int j = 0; j < SPT; j++) {
          const int zz = (int)zzd[j], d = zz >> 16;
          const int ka = c ? kend[krow0 * 64 + d] : 0;
          int cnt = kend[krow1 * 64 + d] - ka;
          const int e0 = reinterpret_cast<const uint16_t *>(rec + NB_REC_OFF)[d] + ka;
          const int zA = (zz & 255) + ka, zB = ((zz >> 8) & 255) - ka;
          uint32_t ep = rec_u + NB_REC_ENT + e0 * 8;
          const uint32_t base = g_u - ((uint32_t)s0 << LOGG);
          uint32_t cA0 = base + plane_off(zA + 1, 4), cB0 = base + plane_off(zB, 4);
          uint32_t cA1 = cA0 + 256 - ((zA + 1) & 1) * 508;
          uint32_t cB1 = cB0 + 252 - (zB & 1) * 508;
          // upward flow over a plane boundary is positive; image k of a row is k * 512 bytes on.
          // q = floor(f V) = high word of f 2^26 by V 2^6
          auto cross = [&](int f, uint32_t rA, uint32_t rB) {
#pragma unroll
            for (int k = 0; k < BS; k++) {
              const int qA = __mulhi(VA[j][k] << (32 - QBITS), f);
              const int qB = __mulhi(VB_[j][k] << (32 - QBITS), f);
              reds_add_s32(rA + 512u * k, VA[j][k] - qA);
              reds_add_s32(rA + 512u * k + (1u << LOGG), qA);
              reds_add_s32(rB + 512u * k, qB - VB_[j][k]);
              reds_add_s32(rB + 512u * k + (1u << LOGG), -qB);
            }
          };
          for (; cnt >= 2; cnt -= 2) {
            int i0, i1, f0, f1;
            lds_ent(ep, i0, f0);
            lds_ent(ep + 8, i1, f1);
            ep += 16;
            cross(f0, cA0 + (i0 << LOGG), cB0 + (i0 << LOGG));
            cross(f1, cA1 + (i1 << LOGG), cB1 + (i1 << LOGG));
            cA0 += 4;
            cA1 += 4;
            cB0 -= 4;
            cB1 -= 4;
          }
          if (cnt) {
            int i0, f0;
            lds_ent(ep, i0, f0);
            cross(f0, cA0 + (i0 << LOGG), cB0 + (i0 << LOGG));
          }
        }
        if (warp == 0) nb_bulk_wait_read<0>();
        __syncthreads();
        const bool last = c == nch - 1;
        if (last && tid == 0) next_job(job);
        // flows -> running sums: this thread's planes z = 2 s and 2 s + 1, SEGL steps
        int rE[SEGL][BS], rO[SEGL][BS], cy[2][BS];
        int *g0 = gacc + seg * SEGL * BS * 128 + s;
#pragma unroll
        for (int v = 0; v < BS; v++) {
          int tE = 0, tO = 0, lp[SEGL];
          if (s == 31)                        // its neighbour above is another warp's
#pragma unroll
            for (int j = 0; j < SEGL; j++) lp[j] = g0[(j * BS + v) * 128 + 1];
          if (s == 63)                        // nothing crosses the top of plane 127
#pragma unroll
            for (int j = 0; j < SEGL; j++) lp[j] = 0;
#pragma unroll
          for (int j = 0; j < SEGL; j++) {
            const int ge = g0[(j * BS + v) * 128], go = g0[(j * BS + v) * 128 + 64];
            int gn = __shfl_down_sync(0xffffffffu, ge, 1);
            if (lane == 31) gn = lp[j];
            tE += ge - go;
            tO += go - gn;
            rE[j][v] = tE;
            rO[j][v] = tO;
          }
          sseg[(seg * 128 + s) * BS + v] = tE;
          sseg[(seg * 128 + 64 + s) * BS + v] = tO;
          if (seg == 0) {                     // the row that spills into the next chunk
            cy[0][v] = g0[(CH * BS + v) * 128];
            cy[1][v] = g0[(CH * BS + v) * 128 + 64];
          }
        }
        float lt[SEGL];
        step_lengths(s0, lt);
        __syncthreads();
        const int *run0 = srun + (c & 1) * 128 * BS;
        int *run1 = srun + ((c & 1) ^ 1) * 128 * BS;
        int bE[BS], bO[BS];
        ldi<BS>(run0 + s * BS, bE);
        ldi<BS>(run0 + (64 + s) * BS, bO);
        for (int x = 0; x < seg; x++) {
          int u[BS], w[BS];
          ldi<BS>(sseg + (x * 128 + s) * BS, u);
          ldi<BS>(sseg + (x * 128 + 64 + s) * BS, w);
#pragma unroll
          for (int v = 0; v < BS; v++) bE[v] += u[v], bO[v] += w[v];
        }
        if (seg == NSEG - 1) {
          int u[BS], w[BS];
#pragma unroll
          for (int v = 0; v < BS; v++) {
            u[v] = bE[v] + rE[SEGL - 1][v];
            w[v] = bO[v] + rO[SEGL - 1][v];
          }
          sti<BS>(run1 + s * BS, u);
          sti<BS>(run1 + (64 + s) * BS, w);
        }
        float ie[BS], io[BS];                 // plane 127 is padding: nothing goes back to it
#pragma unroll
        for (int v = 0; v < BS; v++) {
          ie[v] = inv[v];
          io[v] = s == 63 ? 0.f : ie[v];
        }
        float *o0 = stage + (seg * SEGL * 128 + s) * BS;
#pragma unroll
        for (int j = 0; j < SEGL; j++) {
          int oe[BS], oo[BS];
#pragma unroll
          for (int v = 0; v < BS; v++) {
            oe[v] = __float_as_int((float)(bE[v] + rE[j][v]) * (lt[j] * ie[v]));
            oo[v] = __float_as_int((float)(bO[v] + rO[j][v]) * (lt[j] * io[v]));
            g0[(j * BS + v) * 128] = 0;
            g0[(j * BS + v) * 128 + 64] = 0;
          }
          sti<BS>(reinterpret_cast<int *>(o0) + j * 128 * BS, oe);
          sti<BS>(reinterpret_cast<int *>(o0) + j * 128 * BS + 64 * BS, oo);
        }
        if (seg == 0) {
#pragma unroll
          for (int v = 0; v < BS; v++) {
            g0[v * 128] = last ? 0 : cy[0][v];
            g0[v * 128 + 64] = last ? 0 : cy[1][v];
            g0[(CH * BS + v) * 128] = 0;
            g0[(CH * BS + v) * 128 + 64] = 0;
          }
        }
        nb_fence_proxy_async_smem();
        __syncthreads();
        if (warp == 0) {
          for (int i = lane; i < s1 - s0; i += 32)
            nb_bulk_reduce_add_f32(gb + (size_t)scol[s0 + i] * NB_COLW * BS,
                                   stage + (size_t)i * NB_COLW * BS, NB_COLW * BS * 4);
          nb_bulk_commit();
        }
      }
    }
    __syncthreads();
    q = *snext;
  }
  if (*sflag && tid == 0) nb_set_error(a.err, NB_DEVERR_MBAR_TIMEOUT);
  if (MODE != MODE_FWD && warp == 0) nb_bulk_wait_all<0>();
}

}  // namespace nbw

// nb_walk.cu: the geometry's arguments for `nrep` images, `bs` to a walk; and the launch of one
// mode
nbw::WalkArgs nb_walk_args(const nb_geom *g, const int32_t *subs, int nprj, int span, int nrep,
                           int bs);
int nb_walk_launch(nb_geom *g, const nbw::WalkArgs &a, int mode, int bs, cudaStream_t s);

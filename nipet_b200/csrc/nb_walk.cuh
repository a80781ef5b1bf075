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
// from one plane after another and can exceed what any of them holds.  In the back projection a ray's value is rounded once,
// to 2^-22 of the LOR's largest, its two parts of a crossing sum to it exactly, and at most
// 242 rays meet in a plane, so no sum leaves int32.  A chunk that holds a non-finite (or a
// denormal-small) value is walked step by step in float32 instead, which keeps the value in
// the rays that meet it.
//
// Jobs.  One block per (LOR, image group); a finished block takes over a block that has not
// started (cluster launch control), so LORs of 10 to 404 steps even out over the SMs and the
// next LOR's copies are in flight while one ends (a fixed stride over the LORs left the last
// wave 9% of the SMs' time idle at 4894 LORs).
//
// Measured (B200, 1965 MHz; per call, against the step-by-step walk it replaces): attenuation
// factors of all LORs at span 11 28.0 -> 3.4 ms (chunks without any value are skipped), a
// 4894-LOR emission projection 2.16 -> 0.30 ms, a 5003-LOR span-1 back projection 2.57 ->
// 0.84 ms, a drop-in OSEM iteration 64.4 -> 20.9 ms, 9 images batched 341 -> 163 ms.  Against
// the FP64 oracle the error halves (forward 1.2e-7 -> 5e-8, back 1.5e-7 -> 6e-8 relative L2).
// What bounds it: the shared-memory (LSU) pipe at 79 .. 81% of its wavefronts for one image,
// half of them the crossings' (a warp of 32 pairs spans up to 8 ring differences, whose lanes
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
constexpr int QBITS = NB_REC_QBITS;  // crossing fractions are int32 with this many fraction bits

struct WalkArgs {
  const int32_t *scol;
  const float *st;
  const float4 *hdr;
  const unsigned char *rec;   // crossing schedules (nb_internal.cuh: NB_REC_*)
  const uint32_t *rec_off;    // [naw + 1] start of a LOR's record, in 16-byte units
  const nb_slot *slots;
  int nslots;
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
  static constexpr size_t total = misc_off + 128;
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

// One ray over steps [s0, s1) of a chunk, step by step in float32 (chunks whose values have
// no fixed-point scale).  `ent` points at the ray's crossings of the chunk.
template <int BS>
static __device__ __noinline__ void slow_ray(const float *gimg, const int32_t *col,
                                             const float *st, float tp, int s0, int s1, int z,
                                             int dir, const uint2 *ent, int cnt, bool natural,
                                             float *acc) {
  // (plane 127 reads as zero: the padding slot, or no voxel in the natural order)
  auto vox = [&](const float *c, int z, int k) {
    return !natural ? c[nb_zi(z) * BS + k] : (z < NB_IMZ ? c[z] : 0.f);
  };
  for (int s = s0; s < s1; s++) {
    const float tn = st[s], lt = __fsub_rn(tn, tp);
    const float *c = gimg + (size_t)col[s] * (natural ? NB_IMZ : NB_COLW * BS);
    tp = tn;
    if (cnt > 0 && (int)ent->x == s) {
      const float f = (float)(int)ent->y * (1.f / (1 << QBITS));
      for (int k = 0; k < BS; k++)
        acc[k] = fmaf(f * lt, vox(c, z, k), fmaf((1.f - f) * lt, vox(c, z + dir, k), acc[k]));
      z += dir;
      ent++;
      cnt--;
    } else {
      for (int k = 0; k < BS; k++) acc[k] = fmaf(lt, vox(c, z, k), acc[k]);
    }
  }
}

template <int BS, int CH, int NT, int MODE, int MINB>
__global__ void __launch_bounds__(NT, MINB) k_walk(const WalkArgs a) {
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

    // this thread's slots: start planes of the two rays (8 bits each) and ring difference;
    // the few rays whose start plane rounds away from their group's are listed in the record
    uint32_t zzd[SPT];
    const int nirr = *reinterpret_cast<const uint16_t *>(rec + NB_REC_META);
#pragma unroll
    for (int j = 0; j < SPT; j++) {
      const int sl = slot_of(j);
      zzd[j] = 0u;
      if (sl >= a.nslots) continue;
      const uint32_t zz = __ldg(&a.slots[sl].zzd);
      // the upward ray starts m - 1 planes above its ring's, the downward one as many below
      zzd[j] = zz - (uint32_t)(rec[NB_REC_M + (zz >> 16)] - 1) * 255u;
      for (int x = 0; x < nirr; x++) {
        const char4 e = reinterpret_cast<const char4 *>(rec + NB_REC_IRR)[x];
        if (e.x == (int)(zz >> 16) && 2 * (int)e.y == (int)(zz & 255u))
          zzd[j] += (uint32_t)(e.z ? 256 * (int)e.w : (int)e.w);
      }
    }
    if (tid < 64) sobl[tid] = oblique_s(tid, h.y);
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
            if (lane == 0 && u) atomicMax(&smax[(mrot * NSEG + seg) * BS + v], u);
          }
        }
        __syncthreads();
        unsigned any = 0u;
        bool slow = false;
        const float t0 = s0 ? sst[s0 - 1] : h.x;
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
          // bound < 2^e: scale 2^(29 - e); non-finite, above 2^100 or below 2^-60: step by step
          const int e = (int)(bb >> 23) - 126;
          slow |= bb >= 0x71800000u || (bb != 0u && bb < 0x21800000u);
          scale[k] = bb ? __uint_as_float((uint32_t)(min(max(29 - e, -126), 127) + 127) << 23) : 0.f;
          inv[k] = __uint_as_float((uint32_t)(min(max(e - 29, -126), 127) + 127) << 23);
        }
        // cleared two chunks before its next use: its last readers are one barrier back
        if (tid < NSEG * BS) smax[((mrot + 2) % 3) * NSEG * BS + tid] = 0u;
        mrot = (mrot + 1) % 3;
        if (any == 0u) continue;              // nothing but zeros
        if (!slow) {
          // fixed-point running integrals: within the segment, then the segments before it
          int cE[SEGL][BS], cO[SEGL][BS], tE[BS], tO[BS];
          float sv[BS];
#pragma unroll
          for (int v = 0; v < BS; v++) {
            tE[v] = tO[v] = 0;
            sv[v] = scale[v];
          }
#pragma unroll
          for (int j = 0; j < SEGL; j++) {
#pragma unroll
            for (int v = 0; v < BS; v++) {
              const float w = lt[j] * sv[v];
              cE[j][v] = tE[v];
              cO[j][v] = tO[v];
              tE[v] += __float2int_rn(E[j][v] * w);
              tO[v] += __float2int_rn(O[j][v] * w);
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
          if (slow) {
            const uint2 *ent = reinterpret_cast<const uint2 *>(rec + NB_REC_ENT) + e0;
            slow_ray<BS>(gimg, scol, sst, t0, s0, s1, zA, 1, ent, cnt, natural, FA[j]);
            slow_ray<BS>(gimg, scol, sst, t0, s0, s1, zB, -1, ent, cnt, natural, FB[j]);
            continue;
          }
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
      __syncthreads();   // the walk is done: the table region and the record are free
      if (MODE == MODE_FWD && tid == 0) next_job(job);

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
      float mm[BS];
#pragma unroll
      for (int k = 0; k < BS; k++) mm[k] = 0.f;
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
          mm[k] = fmaxf(mm[k], fmaxf(fabsf(FA[j][k]), fabsf(FB[j][k])));
        }
      }
      const int par = job & 1;
#pragma unroll
      for (int k = 0; k < BS; k++) {
        const unsigned m = __reduce_max_sync(0xffffffffu, __float_as_uint(mm[k]));
        if (lane == 0 && m) atomicMax(&smaxb[par * BS + k], m);
      }
      for (int i = tid; i < 128 * BS; i += NT) srun[i] = 0;
      __syncthreads();
      if (MODE == MODE_OSEM)                  // (the ratios have been read; a barrier follows)
        for (int i = tid; i < (CH + 1) * 32 * BS; i += NT)
          reinterpret_cast<int4 *>(gacc)[i] = make_int4(0, 0, 0, 0);
      float inv[BS];
      int VA[SPT][BS], VB_[SPT][BS];          // the rays' values, integers
      unsigned any = 0u;
#pragma unroll
      for (int k = 0; k < BS; k++) {
        const unsigned mb = smaxb[par * BS + k];
        float sc = 0.f;
        inv[k] = 0.f;
        if (mb != 0u && (mb >> 23) < 255u) {
          const int e = max((int)(mb >> 23) - 126, -96);   // max < 2^e
          sc = __uint_as_float((uint32_t)(FXBITS - e + 127) << 23);
          inv[k] = __uint_as_float((uint32_t)(e - FXBITS + 127) << 23);
          any = 1u;
        }
#pragma unroll
        for (int j = 0; j < SPT; j++) {
          // a NaN, or an infinity (scale 0), becomes 0
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

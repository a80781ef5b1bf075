// nb_geom.cu -- geometry handle: transaxial Siddon tables and per-LOR step lists.
//
// Compiled with -fmad=false: the float arithmetic that decides the crossing order is
// written out operation by operation (reference prj/src/tprj.cu:13-172, sddn_tx), and
// the multiply-adds nvcc contracts in the reference by default are explicit
// __fmaf_rn calls here.  Tables are computed once per handle instead of on every
// projector call (reference prjf.cu:284, prjb.cu:256, recon.cu:349).
#include <math.h>
#include <stdlib.h>
#include <string.h>

#include <algorithm>
#include <map>
#include <tuple>
#include <vector>

#include "nb_axial.cuh"
#include "nb_internal.cuh"

// ---------------------------------------------------------------------------------------
// One thread per LOR: tt[10] and the crossing sequence tv[1807] (reference layout).
// ---------------------------------------------------------------------------------------
__global__ void k_siddon_tx(const float4 *__restrict__ crs, const short2 *__restrict__ s2c,
                            int naw, float *__restrict__ tt, unsigned char *__restrict__ tv) {
  int idx = blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= naw) return;
  short c1 = s2c[idx].x, c2 = s2c[idx].y;
  float4 C1 = crs[c1], C2 = crs[c2];
  // crystal-face centres: float sum, double half, rounded to float (tprj.cu:26-30)
  float cc1x = __double2float_rn(0.5 * (double)__fadd_rn(C1.x, C1.z));
  float cc2x = __double2float_rn(0.5 * (double)__fadd_rn(C2.x, C2.z));
  float cc1y = __double2float_rn(0.5 * (double)__fadd_rn(C1.y, C1.w));
  float cc2y = __double2float_rn(0.5 * (double)__fadd_rn(C2.y, C2.w));
  float ex = __fsub_rn(C1.z, C1.x), ey = __fsub_rn(C1.w, C1.y);
  float px = __double2float_rn(__dadd_rn((double)C1.x, 0.5 * (double)ex));
  float py = __double2float_rn(__dadd_rn((double)C1.y, 0.5 * (double)ey));
  float atx = __fsub_rn(cc2x, cc1x), aty = __fsub_rn(cc2y, cc1y);
  float atn = __fsqrt_rn(__fmaf_rn(atx, atx, __fmul_rn(aty, aty)));
  atx = __fdiv_rn(atx, atn);
  aty = __fdiv_rn(aty, atn);
  // chord through the transaxial FOV circle r^2 = TFOV2 (tprj.cu:53-56)
  float Br = __fmul_rn(2.f, __fmaf_rn(px, atx, __fmul_rn(py, aty)));
  float Cr = __fmul_rn(4.f, __fmaf_rn(py, py, __fmaf_rn(px, px, -NB_TFOV2)));
  float sq = __fsqrt_rn(__fmaf_rn(Br, Br, -Cr));
  float t1 = __double2float_rn(0.5 * (double)__fsub_rn(-Br, sq));
  float t2 = __double2float_rn(0.5 * (double)__fadd_rn(-Br, sq));
  // rows (tprj.cu:60-77)
  float y1 = __fmaf_rn(aty, t1, py);
  float sgy = signbit(aty) ? 1.f : 0.f;
  float cy1 = ceilf(__fdiv_rn(y1, NB_VOXY));
  float lr1 = __fmul_rn(NB_VOXY, __fsub_rn(cy1, sgy));
  int v = (int)__dsub_rn(0.5 * NB_IMY, (double)cy1);
  float y2 = __fmaf_rn(aty, t2, py);
  float lr2 = __fmul_rn(NB_VOXY, __fadd_rn(floorf(__fdiv_rn(y2, NB_VOXY)), sgy));
  // the compiled reference fuses the boundary line into the offset (lr - py becomes
  // fma(SZ_VOXY, c, -py)); lr1/lr2 keep the rounded product in their other uses
  float tr1 = __fdiv_rn(__fmaf_rn(NB_VOXY, __fsub_rn(cy1, sgy), -py), aty);
  float cy2 = __fadd_rn(floorf(__fdiv_rn(y2, NB_VOXY)), sgy);
  float tr2 = __fdiv_rn(__fmaf_rn(NB_VOXY, cy2, -py), aty);
  bool y21 = fabsf(__fsub_rn(y2, y1)) >= NB_VOXY;
  bool lr21 = fabsf(__fsub_rn(lr1, lr2)) < NB_L21;
  int nr = (int)__fadd_rn(__fmul_rn((float)y21, roundf(__fdiv_rn(fabsf(__fsub_rn(lr2, lr1)),
                                                                 NB_VOXY))),
                          (float)lr21);
  float dtr;
  if (nr > 0)
    dtr = __fadd_rn(__fdiv_rn(__fsub_rn(tr2, tr1), (float)nr), __fmul_rn((float)lr21, t2));
  else
    dtr = t2;
  // columns (tprj.cu:80-97); x1 is a double holding a float value
  double x1 = (double)__fmaf_rn(atx, t1, px);
  double sgx = signbit(atx) ? 1.0 : 0.0;
  float lc1 = __double2float_rn(
      __dmul_rn((double)NB_VOXY, __dsub_rn(ceil(__ddiv_rn(x1, (double)NB_VOXY)), sgx)));
  int u = (int)__dadd_rn(0.5 * NB_IMX, floor(__ddiv_rn(x1, (double)NB_VOXY)));
  float x2 = __fmaf_rn(atx, t2, px);
  float lc2 = __fmul_rn(NB_VOXY, __fadd_rn(floorf(__fdiv_rn(x2, NB_VOXY)), (float)sgx));
  float tc1 = __fdiv_rn(__fsub_rn(lc1, px), atx);
  float tc2 = __fdiv_rn(
      __fmaf_rn(NB_VOXY, __fadd_rn(floorf(__fdiv_rn(x2, NB_VOXY)), (float)sgx), -px), atx);
  bool x21 = fabsf(__double2float_rn(__dsub_rn((double)x2, x1))) >= NB_VOXY;
  bool lc21 = fabsf(__fsub_rn(lc1, lc2)) < NB_L21;
  int nc = (int)__fadd_rn(__fmul_rn((float)x21, roundf(__fdiv_rn(fabsf(__fsub_rn(lc2, lc1)),
                                                                 NB_VOXY))),
                          (float)lc21);
  float dtc;
  if (nc > 0)
    dtc = __fadd_rn(__fdiv_rn(__fsub_rn(tc2, tc1), (float)nc), __fmul_rn((float)lc21, t2));
  else
    dtc = t2;

  // crossing sequence (tprj.cu:105-157): 1 = row step, 0 = column step
  float ang = atanf(__fdiv_rn(aty, atx));
  unsigned char *T = tv + (size_t)NB_N_TV * idx;
  T[0] = atx >= 0 ? 2 : 0;
  T[1] = aty >= 0 ? 2 : 0;
  int k = 2;
  if ((ang < NB_TA1) & (ang > NB_TA2)) {
    float tf = tc1, ts = tr1;
    for (int i = 0; i <= nc; i++) {
      int tsin = __fsub_rn(tf, ts) > 0.f;
      if (k < NB_N_TV) T[k] = 1;
      k += tsin;
      ts = __fadd_rn(ts, __fmul_rn(dtr, (float)tsin));
      if (k < NB_N_TV) T[k] = 0;
      k += 1;
      tf = __fadd_rn(tf, dtc);
    }
    if (tr2 > tc2) {
      if (k < NB_N_TV) T[k] = 1;
      k += 1;
    }
  } else {
    float tf = tr1, ts = tc1;
    for (int i = 0; i <= nr; i++) {
      int tsin = __fsub_rn(tf, ts) > 0.f;
      if (k < NB_N_TV) T[k] = 0;
      k += tsin;
      ts = __fadd_rn(ts, __fmul_rn(dtc, (float)tsin));
      if (k < NB_N_TV) T[k] = 1;
      k += 1;
      tf = __fadd_rn(tf, dtr);
    }
    if (tc2 > tr2) {
      if (k < NB_N_TV) T[k] = 0;
      k += 1;
    }
  }
  float *t = tt + (size_t)NB_N_TT * idx;
  t[0] = tr1;
  t[1] = tc1;
  t[2] = dtr;
  t[3] = dtc;
  t[4] = t1;
  t[5] = fminf(tr1, tc1);
  t[6] = t2;
  t[7] = atn;
  t[8] = (float)(u + (v << 9));
  t[9] = (float)k;
}

// ---------------------------------------------------------------------------------------
// One thread per LOR: expand the crossing sequence into the step list the projectors
// stream (the walk of prjf.cu:49-86, done once per geometry instead of per ray).
// ---------------------------------------------------------------------------------------
__global__ void k_expand_steps(const float *__restrict__ tt, const unsigned char *__restrict__ tv,
                               int naw, int32_t *__restrict__ scol, float *__restrict__ st,
                               float4 *__restrict__ hdr, int *err) {
  int idx = blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= naw) return;
  const float *t = tt + (size_t)NB_N_TT * idx;
  const unsigned char *T = tv + (size_t)NB_N_TV * idx;
  int sgna0 = T[0] - 1, sgna1 = T[1] - 1;
  int rbit = T[2] & 1;
  int uvp = (int)t[8];
  int v = uvp >> 9;
  int col = (uvp & 0x1ff) + NB_IMX * v;
  col += !rbit * sgna0;
  col -= rbit * sgna1 * NB_IMX;
  float dtr = t[2], dtc = t[3];
  float trc = __fadd_rn(t[0], __fmul_rn((float)rbit, dtr));
  float tcc = __fadd_rn(t[1], __fmul_rn(dtc, (float)!rbit));
  rbit = T[3] & 1;
  float tn = __fadd_rn(__fmul_rn(trc, (float)rbit), __fmul_rn(tcc, (float)!rbit));
  int K = (int)t[9];
  int n = 0;
  int32_t *sc = scol + (size_t)idx * NB_STEP_STRIDE;
  float *sv = st + (size_t)idx * NB_STEP_STRIDE;
  for (int k = 3; k < K; k++) {
    if (n < NB_STEP_STRIDE) {
      sc[n] = (col >= 0 && col < NB_NCOL) ? col : 0;
      sv[n] = tn;
      if (col < 0 || col >= NB_NCOL) nb_set_error(err, NB_DEVERR_BAD_LOR);
    }
    n++;
    trc = __fadd_rn(trc, __fmul_rn(dtr, (float)rbit));
    tcc = __fadd_rn(tcc, __fmul_rn(dtc, (float)!rbit));
    col += !rbit * sgna0;
    col -= rbit * sgna1 * NB_IMX;
    rbit = (k + 1 < NB_N_TV) ? (T[k + 1] & 1) : 0;
    tn = __fadd_rn(__fmul_rn(trc, (float)rbit), __fmul_rn(tcc, (float)!rbit));
  }
  if (n > NB_STEP_STRIDE) {
    nb_set_error(err, NB_DEVERR_STEP_OVERFLOW);
    n = NB_STEP_STRIDE;
  }
  // pad the tail so that 16-byte bulk copies never read uninitialised entries
  for (int i = n; i < ((n + 3) & ~3) && i < NB_STEP_STRIDE; i++) {
    sc[i] = 0;
    sv[i] = 0.f;
  }
  hdr[idx] = make_float4(t[5], t[7], t[6], __int_as_float(n));
}

// Walks every ray of every LOR once at geometry creation (one block per LOR):
//   out[0]  axial positions outside [0, 127]: the projector indexes shared memory by the plane
//           without clamping.  z = 127 is one plane above the image; it maps to a column's zero
//           padding slot (reads 0, back projections into it are discarded).  In the mMR geometry
//           exactly one ray step reaches it (the last step of rings 59->63 on LOR 24839).
//   out[1]  the longest piece of a walk in cm, as float bits (a crossing that the reference takes
//           a step late, when a ray passes two planes in one, has a negative piece)
//   out[2]  the largest sum of |weight| that the rays of a LOR bring to one plane in one step, as
//           float bits, of the LORs with such crossings; elsewhere every weight is in [0, 1] and
//           at most 242 rays meet in a plane (121 ring differences and directions, of each of
//           which one is in a plane, and one more enters it in the step)
__global__ void __launch_bounds__(256) k_check_walk(const float4 *__restrict__ hdr,
                                                    const float *__restrict__ st,
                                                    const nb_ray *__restrict__ rays, int naw,
                                                    unsigned *out) {
  constexpr int CH = 64;
  __shared__ float acc[CH][128];
  const int lor = blockIdx.x;
  if (lor >= naw) return;
  const float4 h = hdr[lor];
  const int n = __float_as_int(h.w);
  const float *t = st + (size_t)lor * NB_STEP_STRIDE;
  // the walk of a ray; piece(step, plane, length, step's length)
  auto walk = [&](int ray, int end, auto piece) {
    nb_axial A;
    nb_axial_setup(rays[ray], h.y, h.x, h.z, A);
    int w = A.w;
    float tzc = A.tzc, tp = h.x;
    piece(-1, w, 0.f, 0.f);
    for (int k = 0; k < end; k++) {
      const float tn = t[k], lt = __fsub_rn(tn, tp);
      if (tn > tzc) {
        piece(k, w, __fsub_rn(tzc, tp), lt);
        w += A.dir;
        piece(k, w, __fsub_rn(tn, tzc), lt);
        tzc = __fadd_rn(tzc, A.dtz);
      } else {
        piece(k, w, lt, lt);
      }
      tp = tn;
    }
  };
  unsigned nbad = 0;
  float longest = 0.f;
  bool late = false;
  for (int ray = threadIdx.x; ray < NB_NRAYS; ray += blockDim.x)
    walk(ray, n, [&](int, int w, float len, float lt) {
      nbad += w < 0 || w > NB_IMZ;
      longest = fmaxf(longest, fabsf(len));
      late |= fabsf(len) > lt;
    });
  if (nbad) atomicAdd(out, nbad);
  atomicMax(out + 1, __float_as_uint(longest));
  if (__syncthreads_or(nbad) || !__syncthreads_or(late)) return;
  float most = 0.f;
  for (int c = 0; c < n; c += CH) {
    __syncthreads();
    for (int i = threadIdx.x; i < CH * 128; i += blockDim.x) acc[i >> 7][i & 127] = 0.f;
    __syncthreads();
    for (int ray = threadIdx.x; ray < NB_NRAYS; ray += blockDim.x)
      walk(ray, min(n, c + CH), [&](int k, int w, float len, float lt) {
        if (k >= c && lt > 0.f) atomicAdd(&acc[k - c][w], fabsf(len) / lt);
      });
    __syncthreads();
    for (int i = threadIdx.x; i < CH * 128; i += blockDim.x) most = fmaxf(most, acc[i >> 7][i & 127]);
  }
  atomicMax(out + 2, __float_as_uint(most));
}

// ---------------------------------------------------------------------------------------
// Crossing schedules (layout: nb_internal.cuh).  Rays of one ring difference d start two
// planes apart per ring and their crossing parameters are the same floats (ring positions and
// planes are exact multiples of 13/128 cm), so one ray of a difference stands for all: the
// schedule is that ray's own walk (prjf.cu:164-190: at most one crossing a step, the crossing
// parameter advanced by float additions).  What differs between the rays of a difference is
// the start plane where it rounds across a plane boundary (~700 of 2.8e8 rays); those are
// listed with their offset.  Where the first or last boundary of a pair rounds to the next one
// (some pairs of one difference on 18 of the mMR's LORs), its first crossing or their spacing is another float; the
// additions of another spacing drift by up to 1e-4 cm along the walk.  Such pairs get a schedule
// of their own, numbered 61 .. 63.
//
// One block of 64 threads per LOR, thread d for difference d.  FILL = false counts: sizes[lor]
// in 16-byte units; FILL = true writes the records.  err: a schedule or list over capacity.
// ---------------------------------------------------------------------------------------
template <bool FILL>
__global__ void k_sched(const float4 *__restrict__ hdr, const float *__restrict__ st,
                        uint32_t *__restrict__ sizes, const uint32_t *__restrict__ rec_off,
                        unsigned char *__restrict__ rec, int *err) {
  const int lor = blockIdx.x, d = threadIdx.x;
  __shared__ int scnt[64], soff[64], nirr, nalt, alt_d[NB_REC_NALT], alt_r0[NB_REC_NALT];
  const float4 h = hdr[lor];
  const int n = __float_as_int(h.w);
  const float *t = st + (size_t)lor * NB_STEP_STRIDE;
  unsigned char *out = FILL ? rec + (size_t)rec_off[lor] * 16 : nullptr;
  if (d == 0) nirr = nalt = 0;
  __syncthreads();
  int m = 1, rc = 0;
  bool live = d >= 1 && d <= NB_MAXRD && n > 0;
  auto first = [&](int r0, int d) { return nb_first_plane(nb_ring_pair(r0, d, 1), h.y, h.x) - 2 * r0; };
  auto up_ray = [&](int r0, int d, nb_axial &U) { nb_axial_setup(nb_ring_pair(r0, d, 1), h.y, h.x, h.z, U); };
  // do the pairs r0 and r1 of difference d cross at the same floats?
  auto same = [&](int r0, int r1, int d) {
    nb_axial U, V;
    up_ray(r0, d, U);
    up_ray(r1, d, V);
    return first(r0, d) == first(r1, d) && __float_as_int(U.tzc) == __float_as_int(V.tzc) &&
           __float_as_int(U.dtz) == __float_as_int(V.dtz);  // (a single crossing has no spacing: NaN)
  };
  // the pair whose schedule pair r0 of this thread's difference follows, and its number
  auto schedule = [&](int r0, int &id) {
    id = d;
    if (same(r0, rc, d)) return rc;
    for (int x = 0; x < min(nalt, NB_REC_NALT); x++)
      if (alt_d[x] == d && same(r0, alt_r0[x], d)) {
        id = NB_MAXRD + 1 + x;
        return alt_r0[x];
      }
    return -1;
  };
  if (live) {
    // the pair that most agree with (Boyer and Moore's majority vote)
    for (int r0 = 0, votes = 0; r0 + d < NB_NRINGS; r0++) {
      if (votes == 0) rc = r0;
      votes += same(r0, rc, d) ? 1 : -1;
    }
    // pairs that cross at other floats
    int mine = 0, own[NB_REC_NALT];
    for (int r0 = 0; r0 + d < NB_NRINGS; r0++) {
      bool found = same(r0, rc, d);
      for (int x = 0; x < mine; x++) found = found || same(r0, own[x], d);
      if (found) continue;
      const int i = atomicAdd(&nalt, 1);
      if (i >= NB_REC_NALT || mine >= NB_REC_NALT) break;
      own[mine++] = r0;
      alt_d[i] = d;
      alt_r0[i] = r0;
    }
  }
  __syncthreads();
  int dd = d;                                  // ring difference of this thread's schedule
  if (d > NB_MAXRD && d - NB_MAXRD - 1 < min(nalt, NB_REC_NALT)) {
    live = true;
    dd = alt_d[d - NB_MAXRD - 1];
    rc = alt_r0[d - NB_MAXRD - 1];
  }
  nb_axial A;
  A.tzc = A.dtz = 0.f;
  if (live) {
    m = first(rc, dd);
    up_ray(rc, dd, A);
  }
  auto walk = [&](bool fill, int base) {
    int k = 0;
    float tp = h.x, tzc = A.tzc;
    for (int s = 0; s < n; s++) {
      const float tn = t[s];
      if (live && tn > tzc) {
        if (fill) {
          const float lt = __fsub_rn(tn, tp);
          const float f = lt > 0.f ? __fdiv_rn(__fsub_rn(tzc, tp), lt) : 0.f;
          if (!(fabsf(f) < 32.f)) atomicOr(err, 4);  // the fixed-point range
          *reinterpret_cast<int2 *>(out + NB_REC_ENT + 8 * (size_t)(base + k)) =
              make_int2(s, __float2int_rn(ldexpf(f, NB_REC_QBITS)));
        }
        k++;
        tzc = __fadd_rn(tzc, A.dtz);
      }
      tp = tn;
      if (fill && ((s & 7) == 7 || s == n - 1)) out[NB_REC_KEND + (s >> 3) * 64 + d] = (uint8_t)k;
    }
    if (fill)
      for (int r = (n + 7) >> 3; r < NB_STEP_STRIDE / 8; r++)
        out[NB_REC_KEND + r * 64 + d] = (uint8_t)k;
    return k;
  };
  scnt[d] = walk(false, 0);
  __syncthreads();
  if (d == 0) {
    int tot = 0;
    for (int x = 0; x < 64; x++) {
      soff[x] = tot;
      tot += scnt[x];
      if (scnt[x] > 255) atomicOr(err, 1);
    }
    if (tot > NB_REC_MAXENT || nalt > NB_REC_NALT) atomicOr(err, 1);
    if (!FILL) sizes[lor] = (uint32_t)(NB_REC_ENT + ((tot + 1) & ~1) * 8) / 16;
  }
  __syncthreads();
  if (!FILL) return;
  walk(true, soff[d]);
  out[NB_REC_M + d] = (uint8_t)m;
  reinterpret_cast<uint16_t *>(out + NB_REC_OFF)[d] = (uint16_t)soff[d];
  if (live && (m < 1 || m > 255)) atomicOr(err, 1);
  if (d > NB_MAXRD) out[NB_REC_META + 2 + d - NB_MAXRD - 1] = (uint8_t)(live ? dd : 0);
  auto list = [&](int r0, int what, int value) {
    const int i = atomicAdd(&nirr, 1);
    if (i < NB_REC_MAXIRR)
      reinterpret_cast<uchar4 *>(out + NB_REC_IRR)[i] =
          make_uchar4((uint8_t)d, (uint8_t)r0, (uint8_t)what, (uint8_t)(int8_t)value);
  };
  if (live && d <= NB_MAXRD)
    for (int r0 = 0; r0 + d < NB_NRINGS; r0++) {
      nb_axial U, D;
      up_ray(r0, d, U);
      nb_axial_setup(nb_ring_pair(r0, d, 2), h.y, h.x, h.z, D);
      int id;
      const int rs = schedule(r0, id);
      if (rs < 0) {
        atomicOr(err, 1);
        continue;
      }
      if (id != d) list(r0, 2, id);
      const int ms = first(rs, d);
      const int bu = U.w - (2 * r0 + ms - 1), bd = D.w - (2 * (r0 + d) - ms + 1);
      for (int dir = 0; dir < 2; dir++) {
        const int b = dir ? bd : bu;
        if (b == 0) continue;
        if (b < -7 || b > 7) atomicOr(err, 2);
        list(r0, dir, b);
      }
    }
  __syncthreads();
  if (d == 0) {
    if (nirr > NB_REC_MAXIRR) atomicOr(err, 2);
    *reinterpret_cast<uint16_t *>(out + NB_REC_META) = (uint16_t)nirr;
  }
}

// ---------------------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------------------
static void nb_geom_free(nb_geom *g) {
  if (!g) return;
  cudaFree(g->d_scol);
  cudaFree(g->d_st);
  cudaFree(g->d_hdr);
  cudaFree(g->d_tt);
  cudaFree(g->d_rays);
  cudaFree(g->d_rec);
  cudaFree(g->d_rec_off);
  cudaFree(g->d_slots);
  cudaFree(g->d_bin11);
  cudaFree(g->d_scratch128);
  cudaFree(g->d_err);
  cudaFree(g->d_one);
  free(g->h_s2c);
  free(g->h_rays);
  free(g);
}

static int run_tables(nb_geom *g, const float *crs_h, const int16_t *s2c_h, float *d_tt,
                      unsigned char *d_tv) {
  float4 *d_crs = nullptr;
  short2 *d_s2c = nullptr;
  int st = NB_OK;
  cudaError_t e = cudaMalloc(&d_crs, 504 * sizeof(float4));
  if (e == cudaSuccess) e = cudaMalloc(&d_s2c, (size_t)g->naw * sizeof(short2));
  if (e == cudaSuccess)
    e = cudaMemcpy(d_crs, crs_h, 504 * sizeof(float4), cudaMemcpyHostToDevice);
  if (e == cudaSuccess)
    e = cudaMemcpy(d_s2c, s2c_h, (size_t)g->naw * sizeof(short2), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemset(d_tv, 0, (size_t)g->naw * NB_N_TV);
  if (e == cudaSuccess) {
    k_siddon_tx<<<(g->naw + 255) / 256, 256>>>(d_crs, d_s2c, g->naw, d_tt, d_tv);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaDeviceSynchronize();
  if (e != cudaSuccess) st = nb_cuda_fail(e, "siddon tables", __FILE__, __LINE__);
  cudaFree(d_crs);
  cudaFree(d_s2c);
  return st;
}

// Ring of a ring front edge z (cm): ring i starts at (i - 32) * AXR (mmraux.py:365-370)
static int ring_of(float z) {
  const double r = (double)z / (double)NB_RING + 0.5 * NB_NRINGS;
  const long i = lrint(r);
  return fabs(r - (double)i) < 1e-4 ? (int)i : -1;
}

// Slots of a set of rays (those of all ring pairs, or of a reduced range): the direct planes
// two to a slot, then the pairs by ring difference and ring.  False if the rays are not ring
// pairs of the mMR's rings with both directions, once each (ring fronts at (i - 32) * 0.40625 cm,
// differences 1 .. 60).
static bool make_slots(const std::vector<nb_ray> &rays, std::vector<nb_slot> &slots) {
  std::map<std::pair<int, int>, nb_slot> pair;  // (d, r0)
  std::map<int, const nb_ray *> direct;
  std::map<std::pair<int, int>, int> seen;
  for (const nb_ray &R : rays) {
    const int r0 = ring_of(R.r0z), r1 = ring_of(R.r1z);
    if (r0 < 0 || r0 >= NB_NRINGS || R.r0z != (float)(r0 - NB_NRINGS / 2) * NB_RING) return false;
    if (R.kind == 0) {
      if (direct.count(r0)) return false;
      direct[r0] = &R;
      continue;
    }
    if (r1 <= r0 || r1 >= NB_NRINGS || r1 - r0 > NB_MAXRD ||
        R.r1z != (float)(r1 - NB_NRINGS / 2) * NB_RING)
      return false;
    const auto key = std::make_pair(r1 - r0, r0);
    nb_slot &S = pair[key];
    if (seen[key] & R.kind) return false;
    seen[key] |= R.kind;
    S.zzd = (uint32_t)(2 * r0) | (uint32_t)(2 * r1) << 8 | (uint32_t)(r1 - r0) << 16;
    (R.kind == 1 ? S.o11A : S.o11B) = R.out11;
    (R.kind == 1 ? S.o1A : S.o1B) = R.out1;
    (R.kind == 1 ? S.nosA : S.nosB) = R.nos;
  }
  for (const auto &kv : seen)
    if (kv.second != 3) return false;
  std::vector<const nb_ray *> dir;
  for (const auto &kv : direct) dir.push_back(kv.second);
  const size_t half = (dir.size() + 1) / 2;
  slots.clear();
  for (size_t i = 0; i < half; i++) {
    nb_slot S{};
    const nb_ray *A = dir[i], *B = half + i < dir.size() ? dir[half + i] : nullptr;
    S.zzd = (uint32_t)(2 * ring_of(A->r0z)) | (uint32_t)(B ? 2 * ring_of(B->r0z) : 0) << 8;
    S.o11A = A->out11;
    S.o1A = A->out1;
    S.nosA = A->nos;
    S.o11B = B ? B->out11 : -1;
    S.o1B = B ? B->out1 : -1;
    S.nosB = B ? B->nos : 1;
    slots.push_back(S);
  }
  for (const auto &kv : pair) slots.push_back(kv.second);
  return slots.size() <= NB_NSLOT;
}

extern "C" int nb_geom_create(int device, const float *crs, int ncrs, const int16_t *s2c,
                              int naw, const float *li2rng, const int16_t *li2sn,
                              const int16_t *li2sn1, const int8_t *li2nos, int nli2r,
                              nb_geom **out) {
  NB_RANGE("nb_geom_create (Siddon tables, walk checks)");
  NB_REQUIRE(out != nullptr, "nb_geom_create: out is NULL");
  *out = nullptr;
  NB_REQUIRE(crs && s2c && li2rng && li2sn && li2sn1 && li2nos, "nb_geom_create: NULL LUT");
  NB_REQUIRE(ncrs == NB_NCRS, "nb_geom_create: crs must have 504 crystals");
  NB_REQUIRE(naw == NB_AW, "nb_geom_create: s2c must have 68516 LORs");
  NB_REQUIRE(nli2r == NB_NLI2R, "nb_geom_create: li2rng must have 2074 ring pairs");
  int ndev = 0;
  NB_CUDA(cudaGetDeviceCount(&ndev));
  NB_REQUIRE(device >= 0 && device < ndev, "nb_geom_create: invalid device");
  NB_CUDA(cudaSetDevice(device));
  for (int i = 0; i < naw; i++) {
    if (s2c[2 * i] < 0 || s2c[2 * i] >= NB_NCRS || s2c[2 * i + 1] < 0 ||
        s2c[2 * i + 1] >= NB_NCRS) {
      nb_set_error_msg("nb_geom_create: s2c[%d] crystal index out of range", i);
      return NB_ERR_ARG;
    }
  }

  nb_geom *g = (nb_geom *)calloc(1, sizeof(nb_geom));
  if (!g) return NB_ERR_NOMEM;
  g->device = device;
  g->naw = naw;
  cudaDeviceGetAttribute(&g->nsm, cudaDevAttrMultiProcessorCount, device);
  memcpy(g->h_crs, crs, sizeof(g->h_crs));
  g->h_s2c = (int16_t *)malloc(sizeof(int16_t) * 2 * naw);
  memcpy(g->h_s2c, s2c, sizeof(int16_t) * 2 * naw);

  // ray tables (host) -------------------------------------------------------------
  std::vector<nb_ray> rays(NB_NRAYS);
  for (int r = 0; r < NB_NRAYS; r++) {
    int li, kind;
    if (r < NB_NRINGS) {
      li = r;
      kind = 0;
    } else if (r < NB_NRINGS + NB_NOBLQ) {
      li = r;
      kind = 1;
    } else {
      li = r - NB_NOBLQ;
      kind = 2;
    }
    nb_ray R;
    R.r0z = li2rng[2 * li];
    R.r1z = li2rng[2 * li + 1];
    R.out11 = kind == 2 ? li2sn[2 * li + 1] : li2sn[2 * li];
    R.out1 = kind == 2 ? li2sn1[2 * li + 1] : li2sn1[2 * li];
    R.kind = (int8_t)kind;
    R.nos = li2nos[li];
    R.li = (int16_t)li;
    if (R.out11 < 0 || R.out11 >= NB_NSN11 || R.out1 < 0 || R.out1 >= NB_NSN1 || R.nos <= 0) {
      free(g->h_s2c);
      free(g);
      nb_set_error_msg("nb_geom_create: axial LUT entry %d out of range", li);
      return NB_ERR_ARG;
    }
    rays[r] = R;
  }
  std::vector<int16_t> ray11(NB_NSN11 * 8, -1), bin11(NB_NSN11 * 8, -1);  // by ray, by slot
  std::vector<int> cnt11(NB_NSN11, 0), cnt1(NB_NSN1, 0);
  for (int r = 0; r < NB_NRAYS; r++) {
    const int o = rays[r].out11, o1 = rays[r].out1;
    if (cnt11[o] >= 8 || cnt1[o1]++) {
      free(g->h_s2c);
      free(g);
      if (cnt11[o] >= 8)
        nb_set_error_msg("nb_geom_create: more than 8 span-1 planes in span-11 sinogram %d", o);
      else
        nb_set_error_msg("nb_geom_create: span-1 sinogram %d mapped twice", o1);
      return NB_ERR_ARG;
    }
    ray11[o * 8 + cnt11[o]++] = (int16_t)r;
  }
  // rays that are not the mMR's ring pairs go without slots and crossing schedules, through the
  // step-by-step kernel (k_walk_any)
  std::vector<nb_slot> slots;
  if (!make_slots(rays, slots)) slots.clear();
  g->nslots = (int)slots.size();
  std::fill(cnt11.begin(), cnt11.end(), 0);
  for (int r = 0; r < 2 * g->nslots; r++) {
    const int o = r & 1 ? slots[r / 2].o11B : slots[r / 2].o11A;
    if (o >= 0) bin11[o * 8 + cnt11[o]++] = (int16_t)r;
  }

  int st = NB_OK;
  unsigned char *d_tv = nullptr;
  g->h_rays = (nb_ray *)malloc(sizeof(nb_ray) * NB_NRAYS);
  if (!g->h_rays) {
    free(g->h_s2c);
    free(g);
    return NB_ERR_NOMEM;
  }
  memcpy(g->h_rays, rays.data(), sizeof(nb_ray) * NB_NRAYS);
#define ALLOC(p, bytes)                                                                        \
  do {                                                                                         \
    if (cudaMalloc((void **)&(p), (bytes)) != cudaSuccess) {                                   \
      cudaGetLastError();                                                                      \
      nb_set_error_msg("nb_geom_create: cudaMalloc of %zu bytes failed", (size_t)(bytes));      \
      st = NB_ERR_NOMEM;                                                                       \
      goto fail;                                                                               \
    }                                                                                          \
  } while (0)
  ALLOC(g->d_scol, sizeof(int32_t) * (size_t)naw * NB_STEP_STRIDE);
  ALLOC(g->d_st, sizeof(float) * (size_t)naw * NB_STEP_STRIDE);
  ALLOC(g->d_hdr, sizeof(float4) * naw);
  ALLOC(g->d_tt, sizeof(float) * NB_N_TT * (size_t)naw);
  ALLOC(g->d_rays, sizeof(nb_ray) * NB_NRAYS);
  ALLOC(g->d_bin11, sizeof(int16_t) * NB_NSN11 * 8);
  ALLOC(g->d_slots, sizeof(nb_slot) * (g->nslots + 1));
  ALLOC(g->d_rec_off, sizeof(uint32_t) * (naw + 1));
  ALLOC(g->d_scratch128, sizeof(float) * NB_IMG_COL128);
  ALLOC(g->d_err, sizeof(int));
  ALLOC(g->d_one, sizeof(float));
  ALLOC(d_tv, (size_t)naw * NB_N_TV);
#undef ALLOC
  {
    const float one = 1.f;
    if (cudaMemcpy(g->d_one, &one, sizeof(float), cudaMemcpyHostToDevice) != cudaSuccess) {
      cudaGetLastError();
      nb_set_error_msg("nb_geom_create: upload of a constant failed");
      st = NB_ERR_CUDA;
      goto fail;
    }
  }
  if (cudaMemset(g->d_err, 0, sizeof(int)) != cudaSuccess ||
      cudaMemset(g->d_scol, 0, sizeof(int32_t) * (size_t)naw * NB_STEP_STRIDE) != cudaSuccess ||
      cudaMemset(g->d_st, 0, sizeof(float) * (size_t)naw * NB_STEP_STRIDE) != cudaSuccess ||
      cudaMemcpy(g->d_rays, rays.data(), sizeof(nb_ray) * NB_NRAYS, cudaMemcpyHostToDevice) !=
          cudaSuccess ||
      cudaMemcpy(g->d_bin11, bin11.data(), sizeof(int16_t) * NB_NSN11 * 8,
                 cudaMemcpyHostToDevice) != cudaSuccess ||
      cudaMemcpy(g->d_slots, slots.data(), sizeof(nb_slot) * g->nslots,
                 cudaMemcpyHostToDevice) != cudaSuccess) {
    st = nb_cuda_fail(cudaGetLastError(), "nb_geom_create upload", __FILE__, __LINE__);
    goto fail;
  }
  st = run_tables(g, crs, s2c, g->d_tt, d_tv);
  if (st != NB_OK) goto fail;
  k_expand_steps<<<(naw + 255) / 256, 256>>>(g->d_tt, d_tv, naw, g->d_scol, g->d_st, g->d_hdr,
                                             g->d_err);
  if (cudaDeviceSynchronize() != cudaSuccess) {
    st = nb_cuda_fail(cudaGetLastError(), "k_expand_steps", __FILE__, __LINE__);
    goto fail;
  }
  {
    int herr = 0;
    cudaMemcpy(&herr, g->d_err, sizeof(int), cudaMemcpyDeviceToHost);
    if (herr) {
      nb_set_error_msg("nb_geom_create: step expansion reported device error %d", herr);
      st = NB_ERR_DEVICE;
      goto fail;
    }
    // walk check, then the schedules: count, place, fill
    unsigned *d_chk = (unsigned *)d_tv, chk[3] = {0u, 0u, 0u};  // (the tables are expanded)
    cudaError_t e = cudaMemset(d_chk, 0, sizeof(chk));
    if (e == cudaSuccess) {
      k_check_walk<<<naw, 256>>>(g->d_hdr, g->d_st, g->d_rays, naw, d_chk);
      e = cudaMemcpy(chk, d_chk, sizeof(chk), cudaMemcpyDeviceToHost);
    }
    if (e == cudaSuccess && chk[0]) {
      nb_set_error_msg("nb_geom_create: %u ray positions leave the axial FOV", chk[0]);
      st = NB_ERR_DATA;
      goto fail;
    }
    float longest, most;
    memcpy(&longest, &chk[1], sizeof(float));
    memcpy(&most, &chk[2], sizeof(float));
    if (e == cudaSuccess && !(longest < 64.f)) {
      nb_set_error_msg("nb_geom_create: walk segments too long (%g cm)", (double)longest);
      st = NB_ERR_DATA;
      goto fail;
    }
    // a plane's sum of integers below 2^23 each leaves int32 above 255 of them (the mMR: 105.8 where
    // crossings are late, 242 at the most elsewhere)
    if (most > 255.f) g->nslots = 0;
    std::vector<uint32_t> off(naw + 1);
    if (e == cudaSuccess && g->nslots) {
      k_sched<false><<<naw, 64>>>(g->d_hdr, g->d_st, g->d_rec_off, nullptr, nullptr, g->d_err);
      e = cudaMemcpy(off.data(), g->d_rec_off, sizeof(uint32_t) * naw, cudaMemcpyDeviceToHost);
    }
    if (e == cudaSuccess && g->nslots) {
      uint64_t tot = 0;  // 16-byte units: 1.2e8 for the mMR
      for (int i = 0; i <= naw; i++) {
        const uint32_t sz = i < naw ? off[i] : 0;
        off[i] = (uint32_t)tot;
        tot += sz;
      }
      if (tot > 0xffffffffull) {
        nb_set_error_msg("nb_geom_create: crossing schedules too large");
        st = NB_ERR_DATA;
        goto fail;
      }
      if (cudaMalloc((void **)&g->d_rec, (size_t)tot * 16) != cudaSuccess) {
        cudaGetLastError();
        nb_set_error_msg("nb_geom_create: cudaMalloc of %zu bytes failed", (size_t)tot * 16);
        st = NB_ERR_NOMEM;
        goto fail;
      }
      e = cudaMemset(g->d_rec, 0, (size_t)tot * 16);
      if (e == cudaSuccess)
        e = cudaMemcpy(g->d_rec_off, off.data(), sizeof(uint32_t) * (naw + 1),
                       cudaMemcpyHostToDevice);
    }
    if (e == cudaSuccess && g->nslots) {
      k_sched<true><<<naw, 64>>>(g->d_hdr, g->d_st, nullptr, g->d_rec_off, g->d_rec, g->d_err);
      e = cudaMemcpy(&herr, g->d_err, sizeof(int), cudaMemcpyDeviceToHost);
    }
    if (e == cudaSuccess) e = cudaMemset(g->d_err, 0, sizeof(int));
    if (herr) g->nslots = 0;  // schedules over capacity: step by step
    if (e == cudaSuccess && !g->nslots) {
      cudaFree(g->d_rec);
      g->d_rec = nullptr;
      e = cudaMemcpy(g->d_bin11, ray11.data(), sizeof(int16_t) * NB_NSN11 * 8,
                     cudaMemcpyHostToDevice);
    }
    if (e != cudaSuccess) {
      st = nb_cuda_fail(e, "nb_geom_create walk check and schedules", __FILE__, __LINE__);
      goto fail;
    }
  }
  cudaFree(d_tv);
  *out = g;
  return NB_OK;
fail:
  cudaFree(d_tv);
  nb_geom_free(g);
  return st;
}

// Rays of the ring range [rs, re) from the range's axial LUTs, as mmraux.axial_lut builds
// them after mmraux.reduce_rings: li2rng / li2sn1 [nli2r][2], the first re - rs entries
// the direct planes (prjf.cu:33-95 runs them as fprj_drct), the others the oblique pairs,
// whose ring r0 -> r1 ray feeds sinogram li2sn1[.][0] and r1 -> r0 li2sn1[.][1]
// (prjf.cu:98-206).  Each ray must be one of the geometry's rays with both rings in the
// range, and the rays must fill the range's (re - rs)^2 sinograms (4084 for all 64 rings)
// once each; anything else is NB_ERR_ARG (the reference's LUTs of 62- and 63-ring ranges,
// whose ring differences exceed the maximum of 60 without the full-ring correction, end in
// zero entries and fail this check).
extern "C" int nb_rings_create(nb_geom *g, int rs, int re, const float *li2rng,
                               const int16_t *li2sn1, int nli2r, nb_rings **out) {
  NB_REQUIRE(out != nullptr, "nb_rings_create: out is NULL");
  *out = nullptr;
  NB_REQUIRE(g && li2rng && li2sn1, "nb_rings_create: NULL argument");
  NB_REQUIRE(g->h_rays != nullptr, "nb_rings_create: geometry without a ray table");
  NB_REQUIRE(rs >= 0 && rs < re && re <= NB_NRINGS, "nb_rings_create: need 0 <= rs < re <= 64");
  const int n = re - rs;
  const int want_li = n * (n + 1) / 2 - (n == NB_NRINGS ? 6 : 0);
  const int nsino = n * n - (n == NB_NRINGS ? 12 : 0);
  if (nli2r != want_li) {
    nb_set_error_msg("nb_rings_create: %d ring pairs given, the range [%d, %d) has %d", nli2r,
                     rs, re, want_li);
    return NB_ERR_ARG;
  }
  // the geometry's rays by (kind, ring front edges)
  std::map<std::tuple<int, uint32_t, uint32_t>, int> pos;
  for (int r = 0; r < NB_NRAYS; r++) {
    const nb_ray &R = g->h_rays[r];
    uint32_t a, b;
    memcpy(&a, &R.r0z, 4);
    memcpy(&b, &R.r1z, 4);
    pos[std::make_tuple((int)R.kind, a, b)] = r;
  }
  std::vector<nb_ray> sel;
  sel.reserve(nsino);
  for (int li = 0; li < nli2r; li++) {
    const float z0 = li2rng[2 * li], z1 = li2rng[2 * li + 1];
    const int r0 = ring_of(z0), r1 = ring_of(z1);
    if (r0 < rs || r0 >= re || r1 < rs || r1 >= re) {
      nb_set_error_msg("nb_rings_create: ring pair %d (z %g, %g cm) is outside rings [%d, %d)",
                       li, (double)z0, (double)z1, rs, re);
      return NB_ERR_ARG;
    }
    const int nk = li < n ? 1 : 2;
    for (int k = 0; k < nk; k++) {
      const int kind = li < n ? 0 : 1 + k;
      uint32_t a, b;
      memcpy(&a, &z0, 4);
      memcpy(&b, &z1, 4);
      auto it = pos.find(std::make_tuple(kind, a, b));
      if (it == pos.end()) {
        nb_set_error_msg("nb_rings_create: ring pair %d (rings %d, %d) is not a %s ray of the "
                         "geometry", li, r0, r1, kind == 0 ? "direct" : "oblique");
        return NB_ERR_ARG;
      }
      nb_ray R = g->h_rays[it->second];
      R.out1 = li2sn1[2 * li + k];
      R.out11 = 0;  // span 11 does not exist for a reduced range
      sel.push_back(R);
    }
  }
  if ((int)sel.size() != nsino) {
    nb_set_error_msg("nb_rings_create: %zu rays for %d sinograms", sel.size(), nsino);
    return NB_ERR_ARG;
  }
  std::vector<char> used(nsino, 0);
  for (const nb_ray &R : sel) {
    if (R.out1 < 0 || R.out1 >= nsino || used[R.out1]) {
      nb_set_error_msg("nb_rings_create: sinogram %d of the range is out of [0, %d) or mapped "
                       "twice", (int)R.out1, nsino);
      return NB_ERR_ARG;
    }
    used[R.out1] = 1;
  }
  std::vector<nb_slot> slots;
  if (!g->nslots || !make_slots(sel, slots)) slots.clear();  // step by step, as the geometry
  NB_CUDA(cudaSetDevice(g->device));
  nb_rings *rr = (nb_rings *)calloc(1, sizeof(nb_rings));
  if (!rr) return NB_ERR_NOMEM;
  rr->device = g->device;
  rr->rs = rs;
  rr->re = re;
  rr->nrays = nsino;
  rr->vz0 = 2 * rs;
  rr->nvz = 2 * n - 1;
  rr->nslots = (int)slots.size();
  cudaError_t e = cudaMalloc(&rr->d_slots, sizeof(nb_slot) * (slots.size() + 1));
  if (e == cudaSuccess)
    e = cudaMemcpy(rr->d_slots, slots.data(), sizeof(nb_slot) * slots.size(),
                   cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMalloc(&rr->d_rays, sizeof(nb_ray) * nsino);
  if (e == cudaSuccess)
    e = cudaMemcpy(rr->d_rays, sel.data(), sizeof(nb_ray) * nsino, cudaMemcpyHostToDevice);
  if (e != cudaSuccess) {
    cudaFree(rr->d_slots);
    cudaFree(rr->d_rays);
    free(rr);
    return nb_cuda_fail(e, "nb_rings_create upload", __FILE__, __LINE__);
  }
  *out = rr;
  return NB_OK;
}

extern "C" int nb_rings_destroy(nb_rings *rr) {
  if (!rr) return NB_OK;
  cudaSetDevice(rr->device);
  cudaFree(rr->d_slots);
  cudaFree(rr->d_rays);
  free(rr);
  return NB_OK;
}

extern "C" int nb_rings_info(const nb_rings *rr, int *nsino, int *vz0, int *nvz) {
  NB_REQUIRE(rr != nullptr, "nb_rings_info: NULL handle");
  if (nsino) *nsino = rr->nrays;
  if (vz0) *vz0 = rr->vz0;
  if (nvz) *nvz = rr->nvz;
  return NB_OK;
}

extern "C" int nb_geom_destroy(nb_geom *g) {
  if (!g) return NB_OK;
  cudaSetDevice(g->device);
  nb_geom_free(g);
  return NB_OK;
}

extern "C" int nb_geom_tables(nb_geom *g, float *tt, uint8_t *tv) {
  NB_REQUIRE(g && tt && tv, "nb_geom_tables: NULL argument");
  NB_CUDA(cudaSetDevice(g->device));
  float *d_tt = nullptr;
  unsigned char *d_tv = nullptr;
  if (cudaMalloc(&d_tt, sizeof(float) * NB_N_TT * (size_t)g->naw) != cudaSuccess ||
      cudaMalloc(&d_tv, (size_t)g->naw * NB_N_TV) != cudaSuccess) {
    cudaGetLastError();
    cudaFree(d_tt);
    cudaFree(d_tv);
    nb_set_error_msg("nb_geom_tables: cudaMalloc failed");
    return NB_ERR_NOMEM;
  }
  int st = run_tables(g, g->h_crs, g->h_s2c, d_tt, d_tv);
  if (st == NB_OK) {
    cudaError_t e = cudaMemcpy(tt, d_tt, sizeof(float) * NB_N_TT * (size_t)g->naw,
                               cudaMemcpyDeviceToHost);
    if (e == cudaSuccess)
      e = cudaMemcpy(tv, d_tv, (size_t)g->naw * NB_N_TV, cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) st = nb_cuda_fail(e, "nb_geom_tables copy", __FILE__, __LINE__);
  }
  cudaFree(d_tt);
  cudaFree(d_tv);
  return st;
}

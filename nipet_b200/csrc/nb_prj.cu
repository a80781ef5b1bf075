// nb_prj.cu -- projector entry points, layout conversion, OSEM element-wise kernels and
// the sinogram gap kernels.  The projector kernel itself is in nb_walk.cuh.
#include <math.h>

#include <algorithm>

#include "nb_axial.cuh"
#include "nb_internal.cuh"
#include "nb_walk.cuh"

namespace {

// ---------------------------------------------------------------------------------------
// layout conversion and element-wise kernels
// ---------------------------------------------------------------------------------------
// reference [320][320][127] -> col128 and back.  A block moves 16 columns through shared
// memory: the natural side is 16 x 127 contiguous floats, 16-byte aligned, the col128 side 16 x
// 128, whole rows either way (a warp per column took 30 and 24 us for 104 MB).  Measured (B200): 31.7 -> 18.4 and 23.0 ->
// 18.4 us an image, 16 us at 6.65 TB/s.
constexpr int CV = 16;
static_assert(NB_NCOL % CV == 0 && CV * NB_IMZ % 4 == 0, "whole, aligned groups of columns");

__global__ void __launch_bounds__(256) k_to_col128(float *__restrict__ dst,
                                                   const float *__restrict__ src, int ncols) {
  __shared__ __align__(16) float t[CV * NB_IMZ];
  for (int g = blockIdx.x; g < ncols / CV; g += gridDim.x) {
    const float *s = src + (size_t)g * CV * NB_IMZ;
    __syncthreads();
    for (int i = threadIdx.x; i < CV * NB_IMZ / 4; i += 256)
      reinterpret_cast<float4 *>(t)[i] = __ldcs(reinterpret_cast<const float4 *>(s) + i);
    __syncthreads();
    float *d = dst + (size_t)g * CV * NB_COLW;
    for (int i = threadIdx.x; i < CV * NB_COLW; i += 256) {
      const int q = i & 127, z = q < 64 ? 2 * q : 2 * (q - 64) + 1;
      d[i] = z < NB_IMZ ? t[(i >> 7) * NB_IMZ + z] : 0.f;
    }
  }
}

__global__ void __launch_bounds__(256) k_from_col128(float *__restrict__ dst,
                                                     const float *__restrict__ src, int ncols) {
  __shared__ __align__(16) float t[CV * NB_IMZ];
  for (int g = blockIdx.x; g < ncols / CV; g += gridDim.x) {
    const float *s = src + (size_t)g * CV * NB_COLW;
    __syncthreads();
    for (int i = threadIdx.x; i < CV * NB_COLW; i += 256) {
      const int q = i & 127, z = q < 64 ? 2 * q : 2 * (q - 64) + 1;
      if (z < NB_IMZ) t[(i >> 7) * NB_IMZ + z] = __ldcs(s + i);
    }
    __syncthreads();
    float4 *d = reinterpret_cast<float4 *>(dst + (size_t)g * CV * NB_IMZ);
    for (int i = threadIdx.x; i < CV * NB_IMZ / 4; i += 256) d[i] = reinterpret_cast<float4 *>(t)[i];
  }
}

// the same for images that do not start on a 16-byte boundary: a warp per column
__global__ void k_to_col128_any(float *__restrict__ dst, const float *__restrict__ src,
                                int ncols) {
  const int wid = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (wid >= ncols) return;
  const float *s = src + (size_t)wid * NB_IMZ;
  float *d = dst + (size_t)wid * NB_COLW;
  for (int z = lane; z < NB_COLW; z += 32) d[nb_zi(z)] = z < NB_IMZ ? s[z] : 0.f;
}

__global__ void k_from_col128_any(float *__restrict__ dst, const float *__restrict__ src,
                                  int ncols) {
  const int wid = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (wid >= ncols) return;
  const float *s = src + (size_t)wid * NB_COLW;
  float *d = dst + (size_t)wid * NB_IMZ;
  for (int z = lane; z < NB_IMZ; z += 32) d[z] = s[nb_zi(z)];
}

// Images of a reduced ring range hold the axial slab [vz0, vz0 + nvz) only
// ([320][320][nvz], z fastest).  Expand: the slab into a full col128 image, zero elsewhere
// (prjf.cu:19-29 imExpand); reduce: the slab out of a col128 image (prjb.cu:19-29
// imReduce).  One warp per column.
__global__ void k_slab_to_col128(float *__restrict__ dst, const float *__restrict__ src,
                                 int nvz, int vz0) {
  const int wid = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (wid >= NB_NCOL) return;
  const float *s = src + (size_t)wid * nvz;
  float *d = dst + (size_t)wid * NB_COLW;
  for (int z = lane; z < NB_COLW; z += 32) {
    const int zr = z - vz0;
    d[nb_zi(z)] = (z < NB_IMZ && zr >= 0 && zr < nvz) ? s[zr] : 0.f;
  }
}

__global__ void k_col128_to_slab(float *__restrict__ dst, const float *__restrict__ src,
                                 int nvz, int vz0) {
  const int wid = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (wid >= NB_NCOL) return;
  const float *s = src + (size_t)wid * NB_COLW;
  float *d = dst + (size_t)wid * nvz;
  for (int z = lane; z < nvz; z += 32) d[z] = s[nb_zi(vz0 + z)];
}

__global__ void k_osem_rs(float *__restrict__ rs, const float *__restrict__ r,
                          const float *__restrict__ s, const float *__restrict__ an_a,
                          const float *__restrict__ an_n, size_t n) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x) {
    // recon.cu:381-398: rsng += ssng; ansng = asng * nsng; rsng = eldiv0(rsng, ansng)
    const float num = s ? __fadd_rn(r[i], s[i]) : r[i];
    const float an = __fmul_rn(an_a[i], an_n[i]);
    rs[i] = (an > -0.000001f && an < 0.000001f) ? 0.f : __fdiv_rn(num, an);
  }
}

// img = msk ? img * (|sens| < 1e-6 ? 0 : bimg / sens) : 0;  bimg = 0   (recon.cu:493-496)
__global__ void k_osem_update(float4 *__restrict__ img, float4 *__restrict__ bimg,
                              const float4 *__restrict__ sens, const uchar4 *__restrict__ msk,
                              size_t n4) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n4;
       i += (size_t)gridDim.x * blockDim.x) {
    float4 x = img[i], b = bimg[i], s = sens[i];
    uchar4 m = msk[i];
#define UPD(c)                                                                                 \
  {                                                                                            \
    float q = (s.c > -0.000001f && s.c < 0.000001f) ? 0.f : __fdiv_rn(b.c, s.c);               \
    x.c = m.c ? x.c * q : 0.f;                                                                 \
  }
    UPD(x) UPD(y) UPD(z) UPD(w)
#undef UPD
    img[i] = x;
    bimg[i] = make_float4(0.f, 0.f, 0.f, 0.f);
  }
}

// V: voxel reads of a full forward projection, one block per LOR
__global__ void k_count_reads(const float4 *__restrict__ hdr, const float *__restrict__ st,
                              const nb_ray *__restrict__ rays, int naw,
                              unsigned long long *out, unsigned long long *per_lor) {
  const int lor = blockIdx.x;
  if (lor >= naw) return;
  const float4 h = hdr[lor];
  const int n = __float_as_int(h.w);
  // per ray: one read per step, one more at each axial crossing (a +RD/-RD pair of the
  // reference: 2 per step, 4 at a crossing); direct rays never cross
  unsigned long long tot = 0;
  for (int ray = threadIdx.x; ray < NB_NRAYS; ray += blockDim.x) {
    nb_axial A;
    nb_axial_setup(rays[ray], h.y, h.x, h.z, A);
    float tzc = A.tzc;
    tot += n;
    for (int k = 0; k < n; k++) {
      const float tn = st[(size_t)lor * NB_STEP_STRIDE + k];
      if (tn > tzc) {
        tot += 1;
        tzc = __fadd_rn(tzc, A.dtz);
      }
    }
  }
  atomicAdd(out, tot);
  atomicAdd(per_lor + lor, tot);
}

int check_common(nb_geom *g, int nprj, const int32_t *subs, int span) {
  NB_REQUIRE(g != nullptr, "NULL geometry handle");
  NB_REQUIRE(span == 1 || span == 11, "span must be 1 or 11");
  NB_REQUIRE(subs == nullptr || nprj >= 0, "nprj must be >= 0");
  NB_CUDA(cudaSetDevice(g->device));
  return NB_OK;
}

}  // namespace

// ---------------------------------------------------------------------------------------
// C ABI
// ---------------------------------------------------------------------------------------
extern "C" int nb_im_to_col128(float *im128, const float *im, int nimg, void *stream) {
  NB_REQUIRE(im128 && im && nimg > 0, "nb_im_to_col128: bad arguments");
  const int ncols = NB_NCOL * nimg;
  if ((((uintptr_t)im128 | (uintptr_t)im) & 15) == 0)
    k_to_col128<<<std::min(ncols / CV, nb_sms() * 8), 256, 0, (cudaStream_t)stream>>>(
        im128, im, ncols);
  else
    k_to_col128_any<<<(ncols * 32 + 255) / 256, 256, 0, (cudaStream_t)stream>>>(im128, im, ncols);
  NB_CUDA(cudaGetLastError());
  return NB_OK;
}

extern "C" int nb_col128_to_im(float *im, const float *im128, int nimg, void *stream) {
  NB_REQUIRE(im128 && im && nimg > 0, "nb_col128_to_im: bad arguments");
  const int ncols = NB_NCOL * nimg;
  if ((((uintptr_t)im128 | (uintptr_t)im) & 15) == 0)
    k_from_col128<<<std::min(ncols / CV, nb_sms() * 8), 256, 0, (cudaStream_t)stream>>>(
        im, im128, ncols);
  else
    k_from_col128_any<<<(ncols * 32 + 255) / 256, 256, 0, (cudaStream_t)stream>>>(im, im128, ncols);
  NB_CUDA(cudaGetLastError());
  return NB_OK;
}

extern "C" int nb_fprj_col128(nb_geom *g, float *sino, const float *im128, const int32_t *subs,
                              int nprj, int span, int att, void *stream) {
  NB_RANGE("nb_fprj");
  int st = check_common(g, nprj, subs, span);
  if (st) return st;
  NB_REQUIRE(sino && im128, "nb_fprj_col128: NULL sino or image");
  NB_REQUIRE(att == 0 || att == 1, "att must be 0 or 1");
  nbw::WalkArgs a = nb_walk_args(g, subs, nprj, span, 1, 1);
  a.att = att;
  a.img = im128;
  a.sino = sino;
  return nb_walk_launch(g, a, nbw::MODE_FWD, 1, (cudaStream_t)stream);
}

extern "C" int nb_bprj_col128(nb_geom *g, float *im128, const float *sino, const int32_t *subs,
                              int nprj, int span, void *stream) {
  NB_RANGE("nb_bprj");
  int st = check_common(g, nprj, subs, span);
  if (st) return st;
  NB_REQUIRE(sino && im128, "nb_bprj_col128: NULL sino or image");
  nbw::WalkArgs a = nb_walk_args(g, subs, nprj, span, 1, 1);
  a.bimg = im128;
  a.sino_in = sino;
  return nb_walk_launch(g, a, nbw::MODE_BWD, 1, (cudaStream_t)stream);
}

extern "C" int nb_sens_col128(nb_geom *g, float *sens128, const float *an, const int32_t *subs,
                              int nprj, int span, void *stream) {
  NB_RANGE("nb_sens");
  int st = check_common(g, nprj, subs, span);
  if (st) return st;
  NB_REQUIRE(sens128 && an, "nb_sens_col128: NULL image or sinogram");
  NB_CUDA(cudaMemsetAsync(sens128, 0, sizeof(float) * NB_IMG_COL128, (cudaStream_t)stream));
  nbw::WalkArgs a = nb_walk_args(g, subs, nprj, span, 1, 1);
  a.bimg = sens128;
  a.sino_in = an;
  a.in_by_lor = 1;
  return nb_walk_launch(g, a, nbw::MODE_BWD, 1, (cudaStream_t)stream);
}

extern "C" int nb_fprj(nb_geom *g, float *sino, const float *im, const int32_t *subs, int nprj,
                       int span, int att, void *stream) {
  NB_RANGE("nb_fprj");
  int st = check_common(g, nprj, subs, span);
  if (st) return st;
  NB_REQUIRE(sino && im, "nb_fprj: NULL sino or image");
  NB_REQUIRE(att == 0 || att == 1, "att must be 0 or 1");
  // the kernel reads the reference layout's columns as they are (their planes in pairs, two
  // wavefronts a read for one): a conversion pass would take 30 us whatever the LORs, against
  // 1% of the walk of a subset
  nbw::WalkArgs a = nb_walk_args(g, subs, nprj, span, 1, 1);
  a.att = att;
  a.img = im;
  a.natural = 1;
  a.sino = sino;
  return nb_walk_launch(g, a, nbw::MODE_FWD, 1, (cudaStream_t)stream);
}

extern "C" int nb_bprj(nb_geom *g, float *im, const float *sino, const int32_t *subs, int nprj,
                       int span, void *stream) {
  int st = check_common(g, nprj, subs, span);
  if (st) return st;
  NB_REQUIRE(sino && im, "nb_bprj: NULL sino or image");
  NB_CUDA(cudaMemsetAsync(g->d_scratch128, 0, sizeof(float) * NB_IMG_COL128,
                          (cudaStream_t)stream));
  st = nb_bprj_col128(g, g->d_scratch128, sino, subs, nprj, span, stream);
  if (st) return st;
  return nb_col128_to_im(im, g->d_scratch128, 1, stream);
}

// Span-1 projections over a reduced ring range (gpu_fprj / gpu_bprj with Cnt.RNG_STRT /
// RNG_END, prjf.cu:209-320, prjb.cu:190-308): images are the range's axial slab
// [320][320][nvz], sinograms [nprj][nsino] numbered by the range's Michelogram.  The slab
// is expanded into the handle's col128 scratch with zeros elsewhere (as the reference's
// imExpand) and the projector walks only the range's rays.
static int check_rings(nb_geom *g, const nb_rings *rr) {
  NB_REQUIRE(rr != nullptr, "NULL ring-range handle");
  NB_REQUIRE(rr->device == g->device, "ring-range handle and geometry on different devices");
  NB_REQUIRE(rr->vz0 >= 0 && rr->nvz > 0 && rr->vz0 + rr->nvz <= NB_IMZ,
             "ring-range handle with a bad axial slab");
  return NB_OK;
}

extern "C" int nb_fprj_rings(nb_geom *g, const nb_rings *rr, float *sino, const float *im,
                             const int32_t *subs, int nprj, int att, void *stream) {
  NB_RANGE("nb_fprj_rings");
  int st = check_common(g, nprj, subs, 1);
  if (st) return st;
  st = check_rings(g, rr);
  if (st) return st;
  NB_REQUIRE(sino && im, "nb_fprj_rings: NULL sino or image");
  NB_REQUIRE(att == 0 || att == 1, "att must be 0 or 1");
  cudaStream_t s = (cudaStream_t)stream;
  k_slab_to_col128<<<(NB_NCOL * 32 + 255) / 256, 256, 0, s>>>(g->d_scratch128, im, rr->nvz,
                                                               rr->vz0);
  NB_CUDA(cudaGetLastError());
  nbw::WalkArgs a = nb_walk_args(g, subs, nprj, 1, 1, 1);
  a.slots = rr->d_slots;
  a.nslots = rr->nslots;
  a.rays = rr->d_rays;
  a.nrays = rr->nrays;
  a.nout = rr->nrays;
  a.att = att;
  a.img = g->d_scratch128;
  a.sino = sino;
  return nb_walk_launch(g, a, nbw::MODE_FWD, 1, s);
}

extern "C" int nb_bprj_rings(nb_geom *g, const nb_rings *rr, float *im, const float *sino,
                             const int32_t *subs, int nprj, void *stream) {
  NB_RANGE("nb_bprj_rings");
  int st = check_common(g, nprj, subs, 1);
  if (st) return st;
  st = check_rings(g, rr);
  if (st) return st;
  NB_REQUIRE(sino && im, "nb_bprj_rings: NULL sino or image");
  cudaStream_t s = (cudaStream_t)stream;
  NB_CUDA(cudaMemsetAsync(g->d_scratch128, 0, sizeof(float) * NB_IMG_COL128, s));
  nbw::WalkArgs a = nb_walk_args(g, subs, nprj, 1, 1, 1);
  a.slots = rr->d_slots;
  a.nslots = rr->nslots;
  a.rays = rr->d_rays;
  a.nrays = rr->nrays;
  a.nout = rr->nrays;
  a.bimg = g->d_scratch128;
  a.sino_in = sino;
  st = nb_walk_launch(g, a, nbw::MODE_BWD, 1, s);
  if (st) return st;
  k_col128_to_slab<<<(NB_NCOL * 32 + 255) / 256, 256, 0, s>>>(im, g->d_scratch128, rr->nvz,
                                                               rr->vz0);
  NB_CUDA(cudaGetLastError());
  return NB_OK;
}

extern "C" int nb_osem_rs(float *rs, const float *rsng, const float *ssng, const float *asng,
                          const float *nsng, size_t n, void *stream) {
  NB_REQUIRE(rs && rsng && asng && nsng, "nb_osem_rs: NULL argument");
  if (n == 0) return NB_OK;
  k_osem_rs<<<1184, 256, 0, (cudaStream_t)stream>>>(rs, rsng, ssng, asng, nsng, n);
  NB_CUDA(cudaGetLastError());
  return NB_OK;
}

extern "C" int nb_osem_subset(nb_geom *g, float *img128, float *bimg128, const float *sens128,
                              const uint8_t *msk128, const uint16_t *psng, const float *rs,
                              const int32_t *subs, int nprj, void *stream) {
  NB_RANGE("nb_osem_subset");
  int st = check_common(g, nprj, subs, 11);
  if (st) return st;
  NB_REQUIRE(img128 && bimg128 && sens128 && msk128 && psng && rs && subs,
             "nb_osem_subset: NULL argument");
  cudaStream_t s = (cudaStream_t)stream;
  NB_CUDA(cudaMemsetAsync(bimg128, 0, sizeof(float) * NB_IMG_COL128, s));
  nbw::WalkArgs a = nb_walk_args(g, subs, nprj, 11, 1, 1);
  a.img = img128;
  a.bimg = bimg128;
  a.psng = psng;
  a.rs = rs;
  st = nb_walk_launch(g, a, nbw::MODE_OSEM, 1, s);
  if (st) return st;
  const size_t n4 = NB_IMG_COL128 / 4;
  k_osem_update<<<g->nsm * 8, 256, 0, s>>>((float4 *)img128, (float4 *)bimg128,
                                           (const float4 *)sens128, (const uchar4 *)msk128, n4);
  NB_CUDA(cudaGetLastError());
  return NB_OK;
}

extern "C" int nb_psf_col128(float *dst128, const float *src128, const float *krnl,
                             float *tmp128, void *stream);

// One OSEM sub-iteration with resolution modelling (recon.cu:459-497 with krnl[0] >= 0):
// the forward projection sees the PSF-convolved image, the back-projected ratio is
// convolved before the division by the (already convolved) sensitivity.  work128 holds two
// col128 images of scratch.
extern "C" int nb_osem_subset_psf(nb_geom *g, float *img128, float *bimg128,
                                  const float *sens128, const uint8_t *msk128,
                                  const uint16_t *psng, const float *rs, const int32_t *subs,
                                  int nprj, const float *krnl, float *work128, void *stream) {
  NB_RANGE("nb_osem_subset_psf");
  int st = check_common(g, nprj, subs, 11);
  if (st) return st;
  NB_REQUIRE(img128 && bimg128 && sens128 && msk128 && psng && rs && subs && krnl && work128,
             "nb_osem_subset_psf: NULL argument");
  cudaStream_t s = (cudaStream_t)stream;
  float *rm = work128, *tmp = work128 + NB_IMG_COL128;
  st = nb_psf_col128(rm, img128, krnl, tmp, stream);
  if (st) return st;
  NB_CUDA(cudaMemsetAsync(bimg128, 0, sizeof(float) * NB_IMG_COL128, s));
  nbw::WalkArgs a = nb_walk_args(g, subs, nprj, 11, 1, 1);
  a.img = rm;
  a.bimg = bimg128;
  a.psng = psng;
  a.rs = rs;
  st = nb_walk_launch(g, a, nbw::MODE_OSEM, 1, s);
  if (st) return st;
  st = nb_psf_col128(rm, bimg128, krnl, tmp, stream);  // rm: the convolved back projection
  if (st) return st;
  NB_CUDA(cudaMemsetAsync(bimg128, 0, sizeof(float) * NB_IMG_COL128, s));
  const size_t n4 = NB_IMG_COL128 / 4;
  k_osem_update<<<g->nsm * 8, 256, 0, s>>>((float4 *)img128, (float4 *)rm,
                                           (const float4 *)sens128, (const uchar4 *)msk128, n4);
  NB_CUDA(cudaGetLastError());
  return NB_OK;
}

extern "C" int nb_geom_count_reads(nb_geom *g, long long *per_lor, long long *reads) {
  NB_REQUIRE(g && reads, "nb_geom_count_reads: NULL argument");
  NB_CUDA(cudaSetDevice(g->device));
  unsigned long long *d = nullptr;
  NB_CUDA(cudaMalloc(&d, sizeof(unsigned long long) * (1 + (size_t)g->naw)));
  cudaMemset(d, 0, sizeof(unsigned long long) * (1 + (size_t)g->naw));
  k_count_reads<<<g->naw, 128>>>(g->d_hdr, g->d_st, g->d_rays, g->naw, d, d + 1);
  unsigned long long h = 0;
  cudaError_t e = cudaMemcpy(&h, d, sizeof(h), cudaMemcpyDeviceToHost);
  if (e == cudaSuccess && per_lor)
    e = cudaMemcpy(per_lor, d + 1, sizeof(long long) * g->naw, cudaMemcpyDeviceToHost);
  cudaFree(d);
  if (e != cudaSuccess) return nb_cuda_fail(e, "nb_geom_count_reads", __FILE__, __LINE__);
  *reads = (long long)h;
  return NB_OK;
}

// ---------------------------------------------------------------------------------------
// gap removal / insertion (scanner_0.cu:94-105, 158-166)
// ---------------------------------------------------------------------------------------
// Both are transposes between [snno][252 * 344] (a sinogram's bins contiguous) and
// [68516][snno] (a LOR's sinograms contiguous), 32 x 32 through shared memory so that either
// side moves whole 128-byte (16-bit: 64-byte) rows; a thread per element read 4 bytes of every
// sector on the Siemens side.  Measured (B200, us at 837 / 4084
// sinograms): float removal 329 / 4731 -> 272 / 1238, 16-bit 270 / 4000 -> 244 / 1136, insertion
// 1504 / 11600 -> 669 / 4733.
template <typename T, bool REMOVE>
__global__ void __launch_bounds__(256) k_gaps(T *__restrict__ dst, const T *__restrict__ src,
                                              int snno, const int32_t *__restrict__ aw2ali) {
  __shared__ T t[32][33];
  const int x = threadIdx.x & 31, y = threadIdx.x >> 5;
  const int na = (NB_AW + 31) / 32, ns = (snno + 31) / 32;
  for (long b = blockIdx.x; b < (long)na * ns; b += gridDim.x) {
    // neighbouring blocks take neighbouring LORs of the same sinograms (the other order took
    // four times as long at 4084 sinograms)
    const int a0 = (int)(b % na) * 32, i0 = (int)(b / na) * 32;
    __syncthreads();
    if (REMOVE) {
      const int aw = a0 + x;
      const int ali = aw < NB_AW ? aw2ali[aw] : 0;
      for (int r = y; r < 32; r += 8)
        if (aw < NB_AW && i0 + r < snno) t[r][x] = src[(size_t)(i0 + r) * NB_NSBINANG + ali];
      __syncthreads();
      for (int r = y; r < 32; r += 8)
        if (a0 + r < NB_AW && i0 + x < snno) dst[(size_t)(a0 + r) * snno + i0 + x] = t[x][r];
    } else {
      for (int r = y; r < 32; r += 8)
        if (a0 + r < NB_AW && i0 + x < snno) t[r][x] = src[(size_t)(a0 + r) * snno + i0 + x];
      __syncthreads();
      const int aw = a0 + x;
      const int ali = aw < NB_AW ? aw2ali[aw] : 0;
      for (int r = y; r < 32; r += 8)
        if (aw < NB_AW && i0 + r < snno) dst[(size_t)(i0 + r) * NB_NSBINANG + ali] = t[x][r];
    }
  }
}

extern "C" int nb_remgaps(float *sng, const float *sino, int snno, const int32_t *aw2ali,
                          void *stream) {
  NB_RANGE("nb_remgaps");
  NB_REQUIRE(sng && sino && aw2ali && snno > 0, "nb_remgaps: bad arguments");
  k_gaps<float, true><<<nb_sms() * 16, 256, 0, (cudaStream_t)stream>>>(sng, sino, snno, aw2ali);
  NB_CUDA(cudaGetLastError());
  return NB_OK;
}

extern "C" int nb_remgaps_u16(uint16_t *sng, const uint16_t *sino, int snno,
                              const int32_t *aw2ali, void *stream) {
  NB_REQUIRE(sng && sino && aw2ali && snno > 0, "nb_remgaps_u16: bad arguments");
  k_gaps<uint16_t, true><<<nb_sms() * 16, 256, 0, (cudaStream_t)stream>>>(sng, sino, snno, aw2ali);
  NB_CUDA(cudaGetLastError());
  return NB_OK;
}

extern "C" int nb_putgaps(float *sino, const float *sng, int snno, const int32_t *aw2ali,
                          void *stream) {
  NB_RANGE("nb_putgaps");
  NB_REQUIRE(sng && sino && aw2ali && snno > 0, "nb_putgaps: bad arguments");
  NB_CUDA(cudaMemsetAsync(sino, 0, sizeof(float) * (size_t)snno * NB_NSBINANG,
                          (cudaStream_t)stream));
  k_gaps<float, false><<<nb_sms() * 16, 256, 0, (cudaStream_t)stream>>>(sino, sng, snno, aw2ali);
  NB_CUDA(cudaGetLastError());
  return NB_OK;
}

extern "C" int nb_geom_check(nb_geom *g, void *stream) {
  NB_REQUIRE(g != nullptr, "nb_geom_check: NULL handle");
  NB_CUDA(cudaSetDevice(g->device));
  return nb_check_device_flag(g, (cudaStream_t)stream);
}

int nb_check_device_flag(nb_geom *g, cudaStream_t stream) {
  NB_CUDA(cudaStreamSynchronize(stream));
  int h = 0;
  NB_CUDA(cudaMemcpy(&h, g->d_err, sizeof(int), cudaMemcpyDeviceToHost));
  if (h) {
    cudaMemset(g->d_err, 0, sizeof(int));
    nb_set_error_msg("device-side error %d", h);
    return NB_ERR_DEVICE;
  }
  return NB_OK;
}

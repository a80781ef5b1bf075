// nb_batch.cu -- OSEM for many images at once: bootstrap replicates or dynamic frames that
// share the scanner geometry, attenuation, normalisation and sensitivity, each with its
// own prompts and image (the batched configuration of the reference's osem(),
// prj/src/recon.cu:318-497, run for all replicates in one launch per sub-iteration).
//
// Layout: "col128 x Bs" -- images grouped Bs at a time, group g at
// img + g * [320*320][128][Bs]; inside a column the Bs replicate values of a voxel are
// contiguous.  The projector kernel (nb_walk.cuh) takes (LOR, group) jobs, so the LOR's
// crossing schedule and every ray's plane sequence are shared by the Bs images.  Its
// forward-only and backward-only modes are the batched projector pair (nb_fprj_batch /
// nb_bprj_batch).
#include <math.h>

#include "nb_axial.cuh"
#include "nb_internal.cuh"
#include "nb_walk.cuh"

constexpr int NB_MAXREP = 1024;

// ---------------------------------------------------------------------------------------
// layout conversion and the batched image update
// ---------------------------------------------------------------------------------------
namespace {

// [nrep][320*320][127] (reference layout) <-> [ngroups][320*320][128][BS]
__global__ void k_to_batch(float *__restrict__ dst, const float *__restrict__ src, int nrep,
                           int bs) {
  const size_t n = (size_t)nrep * NB_NCOL * NB_COLW;
  for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < n;
       t += (size_t)gridDim.x * blockDim.x) {
    const int z = (int)(t % NB_COLW);
    const size_t rc = t / NB_COLW;
    const int col = (int)(rc % NB_NCOL);
    const int rep = (int)(rc / NB_NCOL);
    const int g = rep / bs, k = rep - g * bs;
    const float v = z < NB_IMZ ? src[((size_t)rep * NB_NCOL + col) * NB_IMZ + z] : 0.f;
    dst[(((size_t)g * NB_NCOL + col) * NB_COLW + nb_zi(z)) * bs + k] = v;
  }
}

// every voxel of the nrep images of the batched layout set to `value`; the padding slot of
// each column (slot 127) and the images padding the last group set to zero
__global__ void k_fill_batch(float *__restrict__ dst, float value, int nrep, int bs,
                             size_t n) {
  for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < n;
       t += (size_t)gridDim.x * blockDim.x) {
    const int k = (int)(t % bs);
    const int slot = (int)((t / bs) % NB_COLW);
    const int g = (int)(t / ((size_t)bs * NB_COLW * NB_NCOL));
    dst[t] = (g * bs + k < nrep && slot != NB_COLW - 1) ? value : 0.f;
  }
}

__global__ void k_from_batch(float *__restrict__ dst, const float *__restrict__ src, int nrep,
                             int bs) {
  const size_t n = (size_t)nrep * NB_NCOL * NB_IMZ;
  for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < n;
       t += (size_t)gridDim.x * blockDim.x) {
    const int z = (int)(t % NB_IMZ);
    const size_t rc = t / NB_IMZ;
    const int col = (int)(rc % NB_NCOL);
    const int rep = (int)(rc / NB_NCOL);
    const int g = rep / bs, k = rep - g * bs;
    dst[t] = src[(((size_t)g * NB_NCOL + col) * NB_COLW + nb_zi(z)) * bs + k];
  }
}

// img = msk ? img * (|sens| < 1e-6 ? 0 : bimg / sens) : 0; bimg = 0  (recon.cu:493-496),
// sens and msk shared by the BS images of a group: one thread per voxel of a group moves
// the group's BS values with one vector access (blockIdx.y strides over the groups)

template <int BS>
__global__ void k_update_batch(float *__restrict__ img, float *__restrict__ bimg,
                               const float *__restrict__ sens, const uint8_t *__restrict__ msk,
                               int ngroups) {
  using V = typename nbw::VecF<BS>::T;
  const size_t nvox = (size_t)NB_NCOL * NB_COLW;
  for (int grp = blockIdx.y; grp < ngroups; grp += gridDim.y) {
    V *gi = reinterpret_cast<V *>(img + (size_t)grp * nvox * BS);
    V *gb = reinterpret_cast<V *>(bimg + (size_t)grp * nvox * BS);
    for (size_t v = blockIdx.x * (size_t)blockDim.x + threadIdx.x; v < nvox;
         v += (size_t)gridDim.x * blockDim.x) {
      const float s = sens[v];
      const bool keep = msk[v] != 0;
      const bool zero_s = s > -0.000001f && s < 0.000001f;
      V x = gi[v];
      const V b = gb[v];
      float *xp = reinterpret_cast<float *>(&x);
      const float *bp = reinterpret_cast<const float *>(&b);
#pragma unroll
      for (int k = 0; k < BS; k++) {
        const float q = zero_s ? 0.f : __fdiv_rn(bp[k], s);
        xp[k] = keep ? xp[k] * q : 0.f;
      }
      gi[v] = x;
      V z;
      float *zp = reinterpret_cast<float *>(&z);
#pragma unroll
      for (int k = 0; k < BS; k++) zp[k] = 0.f;
      gb[v] = z;
    }
  }
}

}  // namespace

extern "C" int nb_to_batch(float *dst, const float *src, int nrep, int bs, void *stream) {
  NB_REQUIRE(dst && src && nrep > 0 && (bs == 1 || bs == 2 || bs == 4),
             "nb_to_batch: bad arguments");
  NB_CUDA(cudaMemsetAsync(dst, 0,
                          sizeof(float) * (size_t)((nrep + bs - 1) / bs) * bs * NB_NCOL * NB_COLW,
                          (cudaStream_t)stream));
  k_to_batch<<<4096, 256, 0, (cudaStream_t)stream>>>(dst, src, nrep, bs);
  NB_CUDA(cudaGetLastError());
  return NB_OK;
}

extern "C" int nb_fill_batch(float *dst, float value, int nrep, int bs, void *stream) {
  NB_REQUIRE(dst && nrep > 0 && (bs == 1 || bs == 2 || bs == 4), "nb_fill_batch: bad arguments");
  const size_t n = (size_t)((nrep + bs - 1) / bs) * bs * NB_NCOL * NB_COLW;
  k_fill_batch<<<4096, 256, 0, (cudaStream_t)stream>>>(dst, value, nrep, bs, n);
  NB_CUDA(cudaGetLastError());
  return NB_OK;
}

extern "C" int nb_from_batch(float *dst, const float *src, int nrep, int bs, void *stream) {
  NB_REQUIRE(dst && src && nrep > 0 && (bs == 1 || bs == 2 || bs == 4),
             "nb_from_batch: bad arguments");
  k_from_batch<<<4096, 256, 0, (cudaStream_t)stream>>>(dst, src, nrep, bs);
  NB_CUDA(cudaGetLastError());
  return NB_OK;
}

extern "C" int nb_osem_batch_subset(nb_geom *g, float *img, float *bimg, const float *sens128,
                                    const uint8_t *msk128, const uint16_t *psng, const float *rs,
                                    const float *rscale, int nrep, int bs, int tile,
                                    int span, const int32_t *subs, int nprj, void *stream) {
  NB_RANGE("nb_osem_batch_subset");
  NB_REQUIRE(g != nullptr, "nb_osem_batch_subset: NULL geometry handle");
  NB_REQUIRE(img && bimg && sens128 && msk128 && psng && rs && rscale && subs,
             "nb_osem_batch_subset: NULL argument");
  NB_REQUIRE(nrep > 0 && nrep <= NB_MAXREP, "nb_osem_batch_subset: nrep out of range");
  NB_REQUIRE(span == 11 || span == 1, "nb_osem_batch_subset: span must be 1 or 11");
  NB_REQUIRE(bs == 1 || bs == 2 || bs == 4, "nb_osem_batch_subset: bs must be 1, 2 or 4");
  // (each width has one kernel shape: the tile is checked and has no effect)
  NB_REQUIRE(tile >= 0 && tile <= 2, "nb_osem_batch_subset: tile must be 0, 1 or 2");
  NB_REQUIRE(nprj > 0, "nb_osem_batch_subset: empty subset");
  NB_CUDA(cudaSetDevice(g->device));
  cudaStream_t s = (cudaStream_t)stream;
  const int ngroups = (nrep + bs - 1) / bs;
  nbw::WalkArgs a = nb_walk_args(g, subs, nprj, span, nrep, bs);
  a.img = img;
  a.bimg = bimg;
  a.psng = psng;
  a.rs = rs;
  a.rscale = rscale;
  const int st = nb_walk_launch(g, a, nbw::MODE_OSEM, bs, s);
  if (st) return st;
  const dim3 ugrid(g->nsm * 4, ngroups < 16 ? ngroups : 16);
  if (bs == 4)
    k_update_batch<4><<<ugrid, 256, 0, s>>>(img, bimg, sens128, msk128, ngroups);
  else if (bs == 2)
    k_update_batch<2><<<ugrid, 256, 0, s>>>(img, bimg, sens128, msk128, ngroups);
  else
    k_update_batch<1><<<ugrid, 256, 0, s>>>(img, bimg, sens128, msk128, ngroups);
  NB_CUDA(cudaGetLastError());
  return NB_OK;
}

extern "C" int nb_psf_col128(float *dst128, const float *src128, const float *krnl,
                             float *tmp128, void *stream);

// One span-1 OSEM sub-iteration of one image (the reference's osem() with Cnt.SPN == 1,
// recon.cu:318-497): the batched kernel with one image per walk, whose layout is the col128
// image itself, then the update; with a PSF kernel (krnl, [3][17], may be NULL) the forward
// projection sees the convolved image and the back projection is convolved before the
// update, as nb_osem_subset_psf does at span 11.  work128: two col128 images (PSF only).
extern "C" int nb_osem_subset_span1(nb_geom *g, float *img128, float *bimg128,
                                    const float *sens128, const uint8_t *msk128,
                                    const uint16_t *psng, const float *rs, const int32_t *subs,
                                    int nprj, const float *krnl, float *work128, void *stream) {
  NB_RANGE("nb_osem_subset_span1");
  NB_REQUIRE(g != nullptr, "nb_osem_subset_span1: NULL geometry handle");
  NB_REQUIRE(img128 && bimg128 && sens128 && msk128 && psng && rs && subs,
             "nb_osem_subset_span1: NULL argument");
  NB_REQUIRE(!krnl || work128, "nb_osem_subset_span1: the PSF needs work128");
  NB_REQUIRE(nprj > 0 && nprj <= g->naw, "nb_osem_subset_span1: bad subset size");
  NB_CUDA(cudaSetDevice(g->device));
  cudaStream_t s = (cudaStream_t)stream;
  float *rm = krnl ? work128 : nullptr, *tmp = krnl ? work128 + NB_IMG_COL128 : nullptr;
  if (krnl) {
    const int st = nb_psf_col128(rm, img128, krnl, tmp, stream);
    if (st) return st;
  }
  NB_CUDA(cudaMemsetAsync(bimg128, 0, sizeof(float) * NB_IMG_COL128, s));
  int st = NB_OK;
  cudaError_t e = cudaSuccess;
  {
    nbw::WalkArgs a = nb_walk_args(g, subs, nprj, 1, 1, 1);
    a.img = krnl ? rm : img128;
    a.bimg = bimg128;
    a.psng = psng;
    a.rs = rs;
    st = nb_walk_launch(g, a, nbw::MODE_OSEM, 1, s);
    if (!st && krnl) st = nb_psf_col128(rm, bimg128, krnl, tmp, stream);
    if (!st) {
      k_update_batch<1><<<dim3(g->nsm * 4, 1), 256, 0, s>>>(img128, krnl ? rm : bimg128,
                                                            sens128, msk128, 1);
      e = cudaGetLastError();
    }
  }
  if (e != cudaSuccess) return nb_cuda_fail(e, "nb_osem_subset_span1", __FILE__, __LINE__);
  return st;
}

extern "C" int nb_fprj_batch(nb_geom *g, float *sino, const float *img, int nrep, int bs,
                             int span, const int32_t *subs, int nprj, void *stream) {
  NB_RANGE("nb_fprj_batch");
  NB_REQUIRE(g != nullptr, "nb_fprj_batch: NULL geometry handle");
  NB_REQUIRE(sino && img, "nb_fprj_batch: NULL argument");
  NB_REQUIRE(nrep > 0 && nrep <= NB_MAXREP, "nb_fprj_batch: nrep out of range");
  NB_REQUIRE(span == 11 || span == 1, "nb_fprj_batch: span must be 1 or 11");
  NB_REQUIRE(bs == 1 || bs == 2 || bs == 4, "nb_fprj_batch: bs must be 1, 2 or 4");
  NB_REQUIRE(nprj > 0 && (subs != nullptr || nprj == g->naw), "nb_fprj_batch: bad subset");
  NB_CUDA(cudaSetDevice(g->device));
  nbw::WalkArgs a = nb_walk_args(g, subs, nprj, span, nrep, bs);
  a.img = img;
  a.sino = sino;
  return nb_walk_launch(g, a, nbw::MODE_FWD, bs, (cudaStream_t)stream);
}

extern "C" int nb_bprj_batch(nb_geom *g, float *bimg, const float *sino, int nrep, int bs,
                             int span, const int32_t *subs, int nprj, void *stream) {
  NB_RANGE("nb_bprj_batch");
  NB_REQUIRE(g != nullptr, "nb_bprj_batch: NULL geometry handle");
  NB_REQUIRE(sino && bimg, "nb_bprj_batch: NULL argument");
  NB_REQUIRE(nrep > 0 && nrep <= NB_MAXREP, "nb_bprj_batch: nrep out of range");
  NB_REQUIRE(span == 11 || span == 1, "nb_bprj_batch: span must be 1 or 11");
  NB_REQUIRE(bs == 1 || bs == 2 || bs == 4, "nb_bprj_batch: bs must be 1, 2 or 4");
  NB_REQUIRE(nprj > 0 && (subs != nullptr || nprj == g->naw), "nb_bprj_batch: bad subset");
  NB_CUDA(cudaSetDevice(g->device));
  nbw::WalkArgs a = nb_walk_args(g, subs, nprj, span, nrep, bs);
  a.bimg = bimg;
  a.sino_in = sino;
  return nb_walk_launch(g, a, nbw::MODE_BWD, bs, (cudaStream_t)stream);
}

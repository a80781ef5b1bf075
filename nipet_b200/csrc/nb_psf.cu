// nb_psf.cu -- resolution modelling: the separable 3-D convolution the reference applies
// inside OSEM when a PSF kernel is given (prj/src/recon.cu:49-216, used at :437-445 on the
// sensitivity images, :463-467 on the current image before the forward projection and
// :487-491 on the back projection), on the col128 image layout.
//
// The reference pads the image to [320][320][128] (z fastest), convolves along z with
// kernel row 0, then along the second image axis (x) with row 1, then along the first (y)
// with row 2, each a 17-tap sum with zeros outside the volume, accumulated tap by tap
// from offset -8 to +8 with fused multiply-adds.  The passes here do the same, in the
// same order and with the same rounding, so the results agree bit for bit; z slot 127
// (the padding) stays zero.
#include <cuda_runtime.h>

#include "nb_internal.cuh"

namespace {

constexpr int R = 8;               // kernel radius (RSZ_PSF_KRNL)
constexpr int KL = 2 * R + 1;      // taps per axis

struct PsfKernel {
  float k[3][KL];  // [0] z, [1] second axis (x), [2] first axis (y)
};

// z pass: one warp per transaxial column, four consecutive planes per lane.  The column is
// put in plane order in shared memory with a zero halo; a lane's 20 inputs are five 16-byte
// reads instead of 17 reads per output.  A warp reads its column before it writes it, so dst
// may be src.  VEC: images that start on an 8-byte boundary move two planes at a time; others,
// which the other two passes take as they are, one.
constexpr int ZW = 8;  // warps per block
template <bool VEC>
__global__ void __launch_bounds__(ZW * 32) k_psf_z(float *dst, const float *src,
                                                   const PsfKernel K) {
  __shared__ __align__(16) float sh[ZW][NB_COLW + 2 * R];
  const int lane = threadIdx.x & 31;
  float *s = sh[threadIdx.x >> 5];
  if (lane < R) {
    s[lane] = 0.f;
    s[R + NB_COLW + lane] = 0.f;
  }
  for (int col = blockIdx.x * ZW + (threadIdx.x >> 5); col < NB_NCOL; col += gridDim.x * ZW) {
    // slot of z: even z at z/2, odd z at 64 + z/2; z = 127 is the zero padding slot
    const float *c = src + (size_t)col * NB_COLW + 2 * lane;
    float2 ev, od;
    if (VEC) {
      ev = *reinterpret_cast<const float2 *>(c);
      od = *reinterpret_cast<const float2 *>(c + 64);
    } else {
      ev = make_float2(c[0], c[1]);
      od = make_float2(c[64], c[65]);
    }
    __syncwarp();
    *reinterpret_cast<float4 *>(s + R + 4 * lane) =
        make_float4(ev.x, od.x, ev.y, lane == 31 ? 0.f : od.y);
    __syncwarp();
    float v[4 + 2 * R], o[4];
#pragma unroll
    for (int i = 0; i < 4 + 2 * R; i += 4)
      *reinterpret_cast<float4 *>(v + i) = *reinterpret_cast<const float4 *>(s + 4 * lane + i);
#pragma unroll
    for (int u = 0; u < 4; u++) {
      float sum = 0.f;
#pragma unroll
      for (int j = -R; j <= R; j++) sum = __fmaf_rn(K.k[0][R - j], v[u + R + j], sum);
      o[u] = sum;
    }
    float *q = dst + (size_t)col * NB_COLW + 2 * lane;
    if (lane == 31) o[3] = 0.f;
    if (VEC) {
      *reinterpret_cast<float2 *>(q) = make_float2(o[0], o[2]);
      *reinterpret_cast<float2 *>(q + 64) = make_float2(o[1], o[3]);
    } else {
      q[0] = o[0];
      q[1] = o[2];
      q[64] = o[1];
      q[65] = o[3];
    }
  }
}

// x / y pass: a thread walks one plane slot along a line of columns (AXIS 1: neighbours along
// x, AXIS 2: along y) with the 17 inputs of an output in registers, so an input is read once
// (a line is cut into SEGN parts, whose halos are read twice: 1.2 reads a column) and nothing
// goes through shared memory, whose 17 reads per output bounded the tiled form.  Measured
// (B200): the three passes 194 -> 78 us, against 48 us to read and write 52 MB three times at
// 6.65 TB/s; the copy back (15 us) is gone, since z works in place.
constexpr int SEGN = 4, SEG = NB_IMX / SEGN;
static_assert(NB_IMX == NB_IMY && SEG * SEGN == NB_IMX, "lines of both axes in whole parts");
template <int AXIS>
__global__ void __launch_bounds__(NB_COLW) k_psf_line(float *__restrict__ dst,
                                                      const float *__restrict__ src,
                                                      const PsfKernel K) {
  constexpr size_t step = (size_t)(AXIS == 1 ? 1 : NB_IMX) * NB_COLW;
  const int line = blockIdx.x / SEGN, p0 = (blockIdx.x - line * SEGN) * SEG;
  const int slot = threadIdx.x;  // 0..127
  const size_t base = (size_t)(AXIS == 1 ? line * NB_IMX : line) * NB_COLW + slot;
  const float *in = src + base;
  float *out = dst + base;
  auto at = [&](int p) { return p >= 0 && p < NB_IMX ? __ldg(in + (size_t)p * step) : 0.f; };
  float w[KL + 8 - 1];  // inputs p - R .. p + R + 7
#pragma unroll
  for (int i = 0; i < KL - 1; i++) w[i] = at(p0 - R + i);
  for (int p = p0; p < p0 + SEG; p += 8) {
#pragma unroll
    for (int u = 0; u < 8; u++) w[KL - 1 + u] = at(p + R + u);
#pragma unroll
    for (int u = 0; u < 8; u++) {
      float sum = 0.f;
#pragma unroll
      for (int j = -R; j <= R; j++) sum = __fmaf_rn(K.k[AXIS][R - j], w[u + R + j], sum);
      out[(size_t)(p + u) * step] = slot == 127 ? 0.f : sum;
    }
#pragma unroll
    for (int i = 0; i < KL - 1; i++) w[i] = w[i + 8];
  }
}
static_assert(SEG % 8 == 0, "outputs in eights");

}  // namespace

extern "C" int nb_psf_col128(float *dst128, const float *src128, const float *krnl,
                             float *tmp128, void *stream) {
  NB_RANGE("nb_psf");
  NB_REQUIRE(dst128 && src128 && krnl && tmp128, "nb_psf_col128: NULL argument");
  NB_REQUIRE(dst128 != tmp128 && src128 != tmp128, "nb_psf_col128: tmp must be its own buffer");
  PsfKernel K;
  for (int a = 0; a < 3; a++)
    for (int i = 0; i < KL; i++) K.k[a][i] = krnl[a * KL + i];
  cudaStream_t s = (cudaStream_t)stream;
  const int nsm = nb_sms();
  // z: src -> dst (dst may be src), x: dst -> tmp, y: tmp -> dst: the reference's order.  Images
  // that overlap otherwise go by way of tmp and are copied at the end
  const uintptr_t us = (uintptr_t)src128, ud = (uintptr_t)dst128;
  const bool apart = us == ud || (us < ud ? ud - us : us - ud) >= sizeof(float) * NB_IMG_COL128;
  float *one = apart ? dst128 : tmp128, *two = apart ? tmp128 : dst128;
  if ((((uintptr_t)one | us) & 7) == 0)
    k_psf_z<true><<<nsm * 8, ZW * 32, 0, s>>>(one, src128, K);
  else
    k_psf_z<false><<<nsm * 8, ZW * 32, 0, s>>>(one, src128, K);
  k_psf_line<1><<<NB_IMY * SEGN, NB_COLW, 0, s>>>(two, one, K);
  k_psf_line<2><<<NB_IMX * SEGN, NB_COLW, 0, s>>>(one, two, K);
  if (!apart)
    NB_CUDA(cudaMemcpyAsync(dst128, tmp128, sizeof(float) * NB_IMG_COL128,
                            cudaMemcpyDeviceToDevice, s));
  NB_CUDA(cudaGetLastError());
  return NB_OK;
}

// nb_walk.cu -- launches of the projector kernel (nb_walk.cuh).
#include <atomic>

#include "nb_walk.cuh"

namespace {

template <int BS, int CH, int NT, int MODE, int MINB>
int launch(nb_geom *g, const nbw::WalkArgs &a, cudaStream_t s) {
  constexpr int NSEG = NT / 64;
  constexpr size_t smem = nbw::WSmem<BS, CH, NSEG>::total;
  static_assert(smem * MINB + 1024 * MINB <= 228 * 1024, "too much shared memory per SM");
  auto *k = nbw::k_walk<BS, CH, NT, MODE, MINB>;
  // the shared-memory opt-in is set once per device and kernel shape; host threads may
  // launch concurrently, so the flags are atomics (setting the attribute twice is harmless)
  static std::atomic<bool> set[64];
  if (!set[g->device & 63].load(std::memory_order_acquire)) {
    NB_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    set[g->device & 63].store(true, std::memory_order_release);
  }
  const long jobs = (long)a.nprj * a.ngroups;
  if (jobs <= 0) return NB_OK;
  NB_REQUIRE(jobs <= 0x7fffffff, "too many LORs times images for one launch");
  k<<<(int)jobs, NT, smem, s>>>(a);
  NB_CUDA(cudaGetLastError());
  return NB_OK;
}

// Kernel shapes <BS, steps per chunk, threads, mode, blocks per SM>, one per width.  One image:
// two blocks of 512 threads at 64 registers.  Two and four images need the registers: 16 warps
// of 128 registers an SM beat 32 of 64, which spill (us per image and 4894 LORs, dense image:
// fused sub-iteration / forward / back):
//   one image     64 steps, 2 x 512 threads  1486 / 701 / 764
//                 64 steps, 2 x 256 threads  1653 / 754 / 825
//                 32 steps, 2 x 512 threads  1681 / 797 / 803
//   two images    32 steps, 2 x 256 threads  1257 / 643 / 628
//                 24 steps, 2 x 256 threads  1342 / 698 / 644
//                 64 steps, 1 x 512 threads  1361 / 661 / 720
//                 24 steps, 2 x 384 threads  1406 / 685 / 675
//   four images   32 steps, 1 x 512 threads  1283 / 690 / 649
//                 24 steps, 1 x 384 threads  1414 / 780 / 681
//                 32 steps, 1 x 256 threads  1460 / 754 / 694
//                 32 steps, 1 x 1024 threads 1727 / 942 / 735
// (timed before weak rays were walked again; the shapes taken now: 1420 / 680 / 760, 1252 / 633 /
// 634 and 1281 / 676 / 659).  The order holds for fused sub-iterations of 600 LORs and of 2 to 8 images, at both spans; at 33
// LORs the two-image shape of 512 threads is the faster one (300 against 349 us), but no subset
// is that small.
template <int MODE> int launch_prj(nb_geom *g, const nbw::WalkArgs &a, int bs, cudaStream_t s) {
  if (bs == 4) return launch<4, 32, 512, MODE, 1>(g, a, s);
  if (bs == 2) return launch<2, 32, 256, MODE, 2>(g, a, s);
  return launch<1, 64, 512, MODE, 2>(g, a, s);
}

// The same three modes for rays that are not the mMR's ring pairs, or whose crossings do not fit
// the schedules: a block per (LOR, image group), its rays step by step in float32 as the reference
// walks them, the image and the back projection in global memory.  Nothing but a hand-made
// geometry comes here: 4894 LORs take 14.0 ms forward and 12.0 back, against 0.7 and 0.8.
constexpr int ANY_NT = 256;
template <int MODE>
__global__ void __launch_bounds__(ANY_NT) k_walk_any(const nbw::WalkArgs a, int bs) {
  extern __shared__ float vals[];             // [nrays][bs]
  const int p = blockIdx.x / a.ngroups, g = blockIdx.x - p * a.ngroups;
  int lor = a.subs ? a.subs[p] : p;
  const bool bad = lor < 0 || lor >= a.naw;
  if (bad) {
    if (threadIdx.x == 0) nb_set_error(a.err, NB_DEVERR_BAD_LOR);
    lor = 0;
  }
  const float4 h = a.hdr[lor];
  const int n = bad ? 0 : __float_as_int(h.w);
  const int32_t *scol = a.scol + (size_t)lor * NB_STEP_STRIDE;
  const float *st = a.st + (size_t)lor * NB_STEP_STRIDE;
  const bool natural = MODE == nbw::MODE_FWD && a.natural != 0;
  const size_t stride = natural ? NB_IMZ : (size_t)NB_COLW * bs;
  const size_t first = (size_t)g * NB_IMG_COL128 * bs;
  auto out_of = [&](const nb_ray &R) { return a.span == 11 ? (int)R.out11 : (int)R.out1; };
  // piece(step, plane, length) of a ray's walk; plane 127 is padding
  auto walk = [&](const nb_axial &A, auto piece) {
    int z = A.w;
    float tp = h.x, tzc = A.tzc;
    for (int s = 0; s < n; s++) {
      const float tn = st[s];
      if (tn > tzc) {
        if (z < NB_IMZ) piece(s, z, __fsub_rn(tzc, tp));
        z += A.dir;
        if (z < NB_IMZ) piece(s, z, __fsub_rn(tn, tzc));
        tzc = __fadd_rn(tzc, A.dtz);
      } else if (z < NB_IMZ) {
        piece(s, z, __fsub_rn(tn, tp));
      }
      tp = tn;
    }
  };
  // ratio of a bin (recon.cu:459-470)
  auto ratio = [&](float v, int o, int k) {
    const int rep = g * bs + k;
    if (rep >= a.nrep) return 0.f;
    const size_t gi = (size_t)lor * a.nout + o;
    const float e = v + a.rscale[rep] * a.rs[gi];
    const float y = (float)a.psng[(size_t)rep * a.naw * a.nout + gi];
    return (e > -0.000001f && e < 0.000001f) ? 0.f : __fdiv_rn(y, e);
  };
  if (MODE != nbw::MODE_BWD) {
    for (int ray = threadIdx.x; ray < a.nrays; ray += ANY_NT) {
      const nb_ray R = a.rays[ray];
      nb_axial A;
      nb_axial_setup(R, h.y, h.x, h.z, A);
      float acc[4] = {0.f, 0.f, 0.f, 0.f};
      walk(A, [&](int s, int z, float len) {
        const float *c = a.img + first + (size_t)scol[s] * stride + (natural ? z : nb_zi(z) * bs);
#pragma unroll
        for (int k = 0; k < 4; k++)
          if (k < bs) acc[k] = fmaf(len, c[k], acc[k]);
      });
#pragma unroll
      for (int k = 0; k < 4; k++) {
        if (k >= bs) break;
        float v = acc[k] * A.s;
        if (MODE == nbw::MODE_FWD && a.att == 1) {
          v = expf(-v);
          if (a.span == 11) v = v / (float)R.nos;
        }
        vals[ray * bs + k] = MODE == nbw::MODE_OSEM && a.span != 11 ? ratio(v, R.out1, k) : v;
        if (MODE == nbw::MODE_FWD && a.span != 11 && g * bs + k < a.nrep)
          a.sino[((size_t)(g * bs + k) * a.nprj + p) * a.nout + R.out1] = v;
      }
    }
    __syncthreads();
    if (a.span == 11)
      for (int x = threadIdx.x; x < a.nout * bs; x += ANY_NT) {
        const int o = x / bs, k = x - o * bs;
        const int16_t *lst = a.bin11 + o * 8;
        float v = 0.f;
        for (int r = 0; r < 8; r++)
          if (lst[r] >= 0) v += vals[lst[r] * bs + k];
        if (MODE == nbw::MODE_OSEM) {
          v = ratio(v, o, k);
          for (int r = 0; r < 8; r++)
            if (lst[r] >= 0) vals[lst[r] * bs + k] = v;
        } else if (g * bs + k < a.nrep) {
          a.sino[((size_t)(g * bs + k) * a.nprj + p) * a.nout + o] = v;
        }
      }
    __syncthreads();
  }
  if (MODE != nbw::MODE_FWD) {
    for (int ray = threadIdx.x; ray < a.nrays; ray += ANY_NT) {
      const nb_ray R = a.rays[ray];
      nb_axial A;
      nb_axial_setup(R, h.y, h.x, h.z, A);
      float v[4] = {0.f, 0.f, 0.f, 0.f};
      bool any = false;
#pragma unroll
      for (int k = 0; k < 4; k++) {
        const int rep = g * bs + k;
        if (k >= bs || rep >= a.nrep) break;
        v[k] = A.s * (MODE == nbw::MODE_OSEM
                          ? vals[ray * bs + k]
                          : a.sino_in[((size_t)rep * a.nprj + (a.in_by_lor ? lor : p)) * a.nout + out_of(R)]);
        any |= v[k] != 0.f;
      }
      if (!any) continue;
      walk(A, [&](int s, int z, float len) {
        if (len == 0.f) return;
        float *c = a.bimg + first + ((size_t)scol[s] * NB_COLW + nb_zi(z)) * bs;
#pragma unroll
        for (int k = 0; k < 4; k++)
          if (k < bs && v[k] != 0.f) atomicAdd(c + k, len * v[k]);
      });
    }
  }
}

template <int MODE> int launch_any(nb_geom *g, const nbw::WalkArgs &a, int bs, cudaStream_t s) {
  const size_t smem = sizeof(float) * (size_t)a.nrays * bs;
  static std::atomic<bool> set[64];
  if (!set[g->device & 63].load(std::memory_order_acquire)) {
    NB_CUDA(cudaFuncSetAttribute(k_walk_any<MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)(sizeof(float) * NB_NRAYS * 4)));
    set[g->device & 63].store(true, std::memory_order_release);
  }
  const long jobs = (long)a.nprj * a.ngroups;
  if (jobs <= 0) return NB_OK;
  NB_REQUIRE(jobs <= 0x7fffffff, "too many LORs times images for one launch");
  k_walk_any<MODE><<<(int)jobs, ANY_NT, smem, s>>>(a, bs);
  NB_CUDA(cudaGetLastError());
  return NB_OK;
}

}  // namespace

int nb_walk_launch(nb_geom *g, const nbw::WalkArgs &a, int mode, int bs, cudaStream_t s) {
  if (a.nslots == 0)
    return mode == nbw::MODE_FWD   ? launch_any<nbw::MODE_FWD>(g, a, bs, s)
           : mode == nbw::MODE_BWD ? launch_any<nbw::MODE_BWD>(g, a, bs, s)
                                   : launch_any<nbw::MODE_OSEM>(g, a, bs, s);
  if (mode == nbw::MODE_FWD) return launch_prj<nbw::MODE_FWD>(g, a, bs, s);
  if (mode == nbw::MODE_BWD) return launch_prj<nbw::MODE_BWD>(g, a, bs, s);
  return launch_prj<nbw::MODE_OSEM>(g, a, bs, s);
}

nbw::WalkArgs nb_walk_args(const nb_geom *g, const int32_t *subs, int nprj, int span, int nrep,
                           int bs) {
  nbw::WalkArgs a{};
  a.scol = g->d_scol;
  a.st = g->d_st;
  a.hdr = g->d_hdr;
  a.rec = g->d_rec;
  a.rec_off = g->d_rec_off;
  a.slots = g->d_slots;
  a.nslots = g->nslots;
  a.rays = g->d_rays;
  a.nrays = NB_NRAYS;
  a.bin11 = g->d_bin11;
  a.subs = subs;
  a.nprj = subs ? nprj : g->naw;
  a.naw = g->naw;
  a.ngroups = (nrep + bs - 1) / bs;
  a.nrep = nrep;
  a.nout = span == 11 ? NB_NSN11 : NB_NSN1;
  a.span = span;
  a.rscale = g->d_one;
  a.err = g->d_err;
  return a;
}

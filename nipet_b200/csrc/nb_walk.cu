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
// The order holds for fused sub-iterations of 600 LORs and of 2 to 8 images, at both spans; at 33
// LORs the two-image shape of 512 threads is the faster one (300 against 349 us), but no subset
// is that small.
template <int MODE> int launch_prj(nb_geom *g, const nbw::WalkArgs &a, int bs, cudaStream_t s) {
  if (bs == 4) return launch<4, 32, 512, MODE, 1>(g, a, s);
  if (bs == 2) return launch<2, 32, 256, MODE, 2>(g, a, s);
  return launch<1, 64, 512, MODE, 2>(g, a, s);
}

}  // namespace

int nb_walk_launch(nb_geom *g, const nbw::WalkArgs &a, int mode, int bs, cudaStream_t s) {
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

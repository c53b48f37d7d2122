// Internal interfaces shared between the translation units of libdpb200.
#pragma once
#include "eval_common.cuh"
#include <algorithm>
#include <cmath>
#include <vector>

namespace dpb {
// The mixed fitting kernel's deep weight ring (1, one CTA per SM) or its shallow
// one (0, two), as timed for launches of this many 128-row tiles; every other
// launch, and all of them at -1, take the rule on sizes.
struct FitShape {
  int deep = -1, tiles = 0;
};
// The 128-row tiles of the fitting over all centre types.
inline int fit_tiles(int ntypes, const int *type_count, int nframes) {
  int n = 0;
  for (int t = 0; t < ntypes; ++t) n += (type_count[t] * nframes + 127) / 128;
  return n;
}
}  // namespace dpb

struct dpb_model {
  dpb::DevModel dm;
  std::vector<void *> allocs;
  // the rest of the newest 8 MB block that small parts of the model are placed in
  char *block = nullptr;
  size_t block_left = 0;
  int device;
  // launch shapes chosen by dpb_md_autotune (they never change results):
  // atoms (warps) per block of the mixed dE/dT kernel, and the mixed fitting
  // kernel's shape
  mutable int dT_warps = 4;
  mutable dpb::FitShape fit;
};

namespace dpb {
// 2^k with x 2^k in (2^13, 2^14] (x > 0; 1 for x = 0 or non-finite), k
// clamped to [-40, 40].
inline float pow2_scale_to_2p14(double x) {
  if (!(x > 0.0) || !std::isfinite(x)) return 1.f;
  int k = 14 - (int)std::ceil(std::log2(x));
  k = std::max(-40, std::min(40, k));
  return std::ldexp(1.f, k);
}
int eval_impl(const dpb_model *m, int precision, const float *pos, const int32_t *perm, int natoms, int nframes,
              const int *type_count, const float *box, const int32_t *nbrs, const int *sel, double *energy,
              float *atom_energy, float *force, double *virial, uint32_t *status, void *workspace,
              size_t ws_bytes, cudaStream_t st, const int32_t *seg = nullptr, int nseg = 0);
int nlist_build_impl(const float *pos, const int32_t *perm, int natoms, int nframes, int ntypes,
                     const int *type_count, const int *sel, const float box[3], const float *ref_box, float rc,
                     int32_t *nbrs, float *ref_pos, int32_t *counts, uint32_t *status, void *workspace,
                     size_t ws_bytes, const unsigned *gate, cudaStream_t stream, const float *dbox = nullptr,
                     int nl_warps = 8);
// Times the mixed dE/dT kernel at 2, 4 and 8 atoms per block on the
// workspace of the last mixed evaluation of NF atoms; *best gets the fastest.
int mixed_tune_dT(const DevModel &M, size_t NF, void *ws, cudaStream_t st, int *best);
// The same on the workspace of the last eval_impl call (F = nframes frames).
int eval_tune_dT(const dpb_model *m, int natoms, int nframes, void *workspace, cudaStream_t st, int *best);
}  // namespace dpb

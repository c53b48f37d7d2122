// Type-sorted positions and the neighbour-row store of the tensor-core
// embedding kernels.
#include "rows.cuh"

namespace dpb {

// Positions in type-sorted order with each atom's frame-local user index:
// posS[f N + k] = (r of atom perm[k] of frame f, perm[k]) - one 16-byte
// gather per neighbour in the mixed embedding kernels.
__global__ void k_pos_sorted(size_t NF, int N, const float *__restrict__ pos, const int32_t *__restrict__ perm,
                             float4 *__restrict__ posS) {
  const size_t g = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (g < NF) {
    const size_t f = g / N;
    const int k = (int)(g - f * N);
    const int src = perm ? perm[k] : k;
    const float *p = pos + (f * N + src) * 3;
    posS[g] = make_float4(p[0], p[1], p[2], __int_as_float(src));
  }
}

// Start of an evaluation: forces, energies, virials and the mixed form's error
// word zeroed in one launch.  (A memset each took 1.4 us and left 2 to 6 us
// between them, also inside a graph: 20 us before the first kernel of 196 us at
// 192 atoms.)
__global__ void k_eval_begin(size_t NF, ForceSum *__restrict__ F4, size_t nE, double *__restrict__ energy,
                             double *__restrict__ virial, int *__restrict__ err) {
  const size_t g = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (g < NF) F4[g] = ForceSum{0.0, 0.0, 0.0, 0.0};
  if (g < nE) energy[g] = 0.0;
  if (g < 9 * nE) virial[g] = 0.0;
  if (err && g == 0) *err = 0;
}

int launch_eval_begin(size_t NF, ForceSum *F4, size_t nE, double *energy, double *virial, int *err, cudaStream_t st) {
  const size_t n = std::max(NF, 9 * nE);
  k_eval_begin<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(NF, F4, nE, energy, virial, err);
  count_launch();
  DPB_LAUNCH_CHECK();
  return DPB_OK;
}

int launch_pos_sorted(const SysDesc &D, const float *pos, const int32_t *perm, float4 *posS,
                             cudaStream_t st) {
  const size_t NF = (size_t)D.N * D.F;
  k_pos_sorted<<<(unsigned)((NF + 255) / 256), 256, 0, st>>>(NF, D.N, pos, perm, posS);
  count_launch();
  DPB_LAUNCH_CHECK();
  return DPB_OK;
}

// One warp per (block of ba centre atoms, neighbour type tj), every centre type
// in one launch,
// kRowsCpt rounds of 32 candidates (atom slot, list slot) at a time in
// candidate order: all of their list entries are loaded, then all of their
// neighbour positions gathered from posS, before any is used (the chain is
// two dependent loads per round); the nearest-image displacement and keep
// test are those of mix_compact_round (same arithmetic, so the same rows),
// and the kept rows are appended round by round with a ballot.  Blocks
// outside the store (several images) are left to the embedding kernels' own
// compaction.
constexpr int kRowsCpt = 4;

__global__ void __launch_bounds__(256) k_rows(DevModel M, SysDesc D, int ba, const float4 *__restrict__ posS,
                                                 const float *__restrict__ box, const int32_t *__restrict__ nbrs,
                                                 float4 *__restrict__ rows_g, int *__restrict__ rcnt) {
  const int lane = threadIdx.x & 31;
  const int wg = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  const int blk = wg / D.ntypes, tj = wg - blk * D.ntypes;
  if (blk >= blocks_total(D, ba)) return;
  const BlkPos bp = block_pos(D, ba, blk);
  const int f = bp.f, nb = bp.nb;
  const size_t g0 = bp.g0;
  const size_t frame_base = (size_t)f * D.N;
  const int bs = box_slot(D, g0, f);
  const float3 L = make_float3(box[bs * 3], box[bs * 3 + 1], box[bs * 3 + 2]);
  const int3 ni = image_range(L, M.rcut);
  if (!row_store_covers(D, rows_g, (2 * ni.x + 1) * (2 * ni.y + 1) * (2 * ni.z + 1))) return;
  const float3 inv_l = make_float3(1.f / L.x, 1.f / L.y, 1.f / L.z);
  const float rk = M.rcut + 1e-3f, rk2 = rk * rk;
  const int sel = D.sel[tj], cnt_j = D.offs[tj + 1] - D.offs[tj], total = nb * sel;
  const int col = D.col[tj], jbase = D.offs[tj];
  // the block's centre positions, one per lane
  const float4 cl = lane < nb ? posS[g0 + lane] : make_float4(0.f, 0.f, 0.f, 0.f);
  float4 *out = rows_g + g0 * kRowStoreCap + (size_t)nb * col;
  int n = 0;
  for (int base = 0; base < total; base += 32 * kRowsCpt) {
    int idx[kRowsCpt], slot[kRowsCpt];
#pragma unroll
    for (int k = 0; k < kRowsCpt; ++k) {
      const int p = base + 32 * k + lane;
      slot[k] = p / sel;
      idx[k] = p < total ? nbrs[(g0 + slot[k]) * D.S + col + (p - slot[k] * sel)] & DPB_NBR_INDEX_MASK : cnt_j;
    }
    float4 q[kRowsCpt];
#pragma unroll
    for (int k = 0; k < kRowsCpt; ++k)
      q[k] = idx[k] < cnt_j ? posS[frame_base + jbase + idx[k]] : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int k = 0; k < kRowsCpt; ++k) {
      const int sl = min(slot[k], kBlkAtoms - 1);
      const float cx = __shfl_sync(0xffffffffu, cl.x, sl), cy = __shfl_sync(0xffffffffu, cl.y, sl),
                  cz = __shfl_sync(0xffffffffu, cl.z, sl);
      float4 rv = make_float4(0.f, 0.f, 0.f, 0.f);
      bool keep = false;
      if (idx[k] < cnt_j) {
        const float dx = q[k].x - cx, dy = q[k].y - cy, dz = q[k].z - cz;
        const float ax = fmaf(-L.x, rintf(dx * inv_l.x), dx), ay = fmaf(-L.y, rintf(dy * inv_l.y), dy),
                    az = fmaf(-L.z, rintf(dz * inv_l.z), dz);
        if (ax * ax + ay * ay + az * az < rk2) {
          keep = true;
          rv = make_float4(ax, ay, az, __int_as_float((__float_as_int(q[k].w) << 3) | slot[k]));
        }
      }
      const unsigned m = __ballot_sync(0xffffffffu, keep);
      if (keep) out[n + __popc(m & ((1u << lane) - 1u))] = rv;
      n += __popc(m);
    }
  }
  if (lane == 0) rcnt[g0 * M.ntypes + tj] = n;
}

int launch_rows(const DevModel &M, const SysDesc &D, int ba, const float4 *posS, const float *box,
                const int32_t *nbrs, float4 *rows, int *rcnt, cudaStream_t st) {
  const size_t warps = (size_t)blocks_total(D, ba) * D.ntypes;
  if (!warps) return DPB_OK;
  k_rows<<<(unsigned)((warps + 7) / 8), 256, 0, st>>>(M, D, ba, posS, box, nbrs, rows, rcnt);
  count_launch();
  DPB_LAUNCH_CHECK();
  return DPB_OK;
}

}  // namespace dpb

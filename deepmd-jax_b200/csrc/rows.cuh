// Blocks of centre atoms and their compacted neighbour rows: the row store, its
// streaming, and the in-kernel compaction, shared by the tensor-core embedding
// kernels of both forms.
#pragma once
#include "internal.cuh"
#include "tc.cuh"

namespace dpb {

constexpr int kBlkAtoms = 8;    // centre atoms per block

__host__ __device__ constexpr int round1k(int x) { return (x + 1023) / 1024 * 1024; }

// Bounded wait on the block's MMA barrier, made uniform across the block.
#define MIX_WAIT()                                  \
  do {                                              \
    const bool w_ = tc::mbar_wait(&mbar, ph);       \
    ph ^= 1;                                        \
    ok = __syncthreads_and(w_ && ok) != 0;          \
    tc::fence_after_sync();                         \
  } while (0)

// One block of up to `ba` consecutive centre atoms of one type and frame:
// blocks are numbered type after type, frame after frame within a type.
struct BlkPos {
  int ti, f, nb;  // centre type, frame, atoms of the block
  int first;      // number of the type's first block
  size_t g0;      // its first atom (f * N + sorted index)
};
__host__ __device__ __forceinline__ int blocks_of_type(const SysDesc &D, int ti, int ba) {
  return (D.offs[ti + 1] - D.offs[ti] + ba - 1) / ba * D.F;
}
__host__ __device__ __forceinline__ int blocks_total(const SysDesc &D, int ba) {
  int n = 0;
  for (int t = 0; t < D.ntypes; ++t) n += blocks_of_type(D, t, ba);
  return n;
}
__device__ __forceinline__ BlkPos block_pos(const SysDesc &D, int ba, int blk) {
  BlkPos b;
  b.ti = b.first = 0;
  int n = blocks_of_type(D, 0, ba);
#pragma unroll
  for (int t = 1; t < kMaxTypes; ++t)
    if (t < D.ntypes && b.ti == t - 1 && blk >= n) {
      blk -= n;
      b.first += n;
      b.ti = t;
      n = blocks_of_type(D, t, ba);
    }
  const int cnt = D.offs[b.ti + 1] - D.offs[b.ti], nbpf = (cnt + ba - 1) / ba;
  b.f = blk / nbpf;
  const int a0 = (blk - b.f * nbpf) * ba;
  b.nb = min(ba, cnt - a0);
  b.g0 = (size_t)b.f * D.N + D.offs[b.ti] + a0;
  return b;
}

// L2 prefetch of [base, base + bytes), one line per thread and step (the
// persistent CTAs issue it for their next block while working on this one).
__device__ __forceinline__ void prefetch_range_l2(const void *base, size_t bytes) {
  const char *b = static_cast<const char *>(base);
  for (size_t o = (size_t)threadIdx.x * 128; o < bytes; o += (size_t)blockDim.x * 128) tc::prefetch_l2(b + o);
}
// One round of compaction over CPT * blockDim candidates (atom slot,
// neighbour slot, image) of the block for neighbour type tj: thread t takes
// the CPT consecutive candidates base + t * CPT + k, issues all of their
// gathers (neighbour index, then position and user index from posS) before
// using any, and the
// kept rows are appended to rowbuf in candidate order (so rows stay sorted by
// atom slot) as (x, y, z, packed), packed = (neighbour user index << 3) | slot.
// With one image per pair (nim == 1, boxes wider than 2 rcut) the row's
// displacement is the nearest image d - L rint(d / L), which equals the
// reference's (d - L/2) mod L - L/2 (utils.py:24-26) up to rounding (the mixed
// form is held to a tolerance, not to bits), and the keep test is |x| <
// rcut + 1e-3 A: every row with s(r) != 0 is kept, and a kept row with
// s(r) = 0 adds exact zeros (R~ = 0, ds/dr = 0).  With several images the
// reference's displacement and s(r) decide.  The unread rows [rowstart, rowcount) of earlier rounds (fewer than
// 128) are first moved to the front.
template <int CPT>
__device__ __forceinline__ void mix_compact_round(const SysDesc &D, const DevModel &M, int tj, int base, int total,
                                                  int per_atom, int nim, int3 ni, float3 L, size_t g0,
                                                  size_t frame_base, const float3 *ri_s,
                                                  const float4 *__restrict__ posS, const int32_t *nbrs, float4 *rowbuf,
                                                  int *wcnt, int &rowstart, int &rowcount) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (rowstart > 0) {
    const int rem = rowcount - rowstart;  // < 128 <= blockDim
    float4 carry = make_float4(0.f, 0.f, 0.f, 0.f);
    if (tid < rem) carry = rowbuf[rowstart + tid];
    __syncthreads();
    if (tid < rem) rowbuf[tid] = carry;
    rowstart = 0;
    rowcount = rem;
  }
  const int cnt_j = D.offs[tj + 1] - D.offs[tj];
  const int p0 = base + tid * CPT;
  int idx[CPT], slotk[CPT], mimgk[CPT];
  int slot = p0 / per_atom, rem = p0 - slot * per_atom;  // advanced incrementally below
#pragma unroll
  for (int k = 0; k < CPT; ++k) {
    const int p = p0 + k;
    idx[k] = cnt_j;
    slotk[k] = 0;
    mimgk[k] = 0;
    if (p < total) {
      const int sidx = nim == 1 ? rem : rem / nim;
      slotk[k] = slot;
      mimgk[k] = rem - sidx * nim;
      idx[k] = nbrs[(g0 + slot) * D.S + D.col[tj] + sidx] & DPB_NBR_INDEX_MASK;
    }
    if (++rem == per_atom) {
      rem = 0;
      ++slot;
    }
  }
  int src[CPT];
  float3 pj[CPT];
#pragma unroll
  for (int k = 0; k < CPT; ++k) {
    src[k] = -1;
    pj[k] = make_float3(0.f, 0.f, 0.f);
    if (idx[k] < cnt_j) {
      const float4 q = posS[frame_base + D.offs[tj] + idx[k]];
      pj[k] = make_float3(q.x, q.y, q.z);
      src[k] = __float_as_int(q.w);
    }
  }
  float4 rv[CPT];
  unsigned keep = 0;
  if (nim == 1) {
    const float3 inv_l = make_float3(1.f / L.x, 1.f / L.y, 1.f / L.z);
    const float rk = M.rcut + 1e-3f, rk2 = rk * rk;
#pragma unroll
    for (int k = 0; k < CPT; ++k) {
      rv[k] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (src[k] >= 0) {
        const float3 ri = ri_s[slotk[k]];
        const float dx = pj[k].x - ri.x, dy = pj[k].y - ri.y, dz = pj[k].z - ri.z;
        const float ax = fmaf(-L.x, rintf(dx * inv_l.x), dx), ay = fmaf(-L.y, rintf(dy * inv_l.y), dy),
                    az = fmaf(-L.z, rintf(dz * inv_l.z), dz);
        if (ax * ax + ay * ay + az * az < rk2) {
          keep |= 1u << k;
          rv[k] = make_float4(ax, ay, az, __int_as_float((src[k] << 3) | slotk[k]));
        }
      }
    }
  } else {
#pragma unroll
    for (int k = 0; k < CPT; ++k) {
      rv[k] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (src[k] >= 0) {
        const float3 x = rel_coord(ri_s[slotk[k]], pj[k], L, ni, mimgk[k]);
        RowGeom gm;
        row_geom(x, M.rcut, gm);
        if (gm.s != 0.f) {
          keep |= 1u << k;
          rv[k] = make_float4(x.x, x.y, x.z, __int_as_float((src[k] << 3) | slotk[k]));
        }
      }
    }
  }
  // block-wide exclusive scan of the per-thread counts
  const int c = __popc(keep);
  int incl = c;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int t = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += t;
  }
  if (lane == 31) wcnt[warp] = incl;
  __syncthreads();
  int off = 0, tot = 0;
  for (int w = 0; w < (int)(blockDim.x >> 5); ++w) {
    if (w < warp) off += wcnt[w];
    tot += wcnt[w];
  }
  int o = rowcount + off + incl - c;
#pragma unroll
  for (int k = 0; k < CPT; ++k)
    if (keep >> k & 1u) rowbuf[o++] = rv[k];
  rowcount += tot;
  __syncthreads();
}

// Row store of list mode (one image per pair, boxes wider than 2 rcut):
// k_rows compacts the neighbour rows of every block of ba centre atoms (8 in
// the mixed form; 1, 2 or 4 in the FP32 form) and neighbour type once per
// evaluation, rows of the block of first atom g0 (nb atoms) and type tj at
// rows_g + g0 * kRowStoreCap + nb * col[tj] (in candidate order, so sorted by
// atom slot, as mix_compact_round leaves them), their count at rcnt[g0 *
// ntypes + tj].  The forward and the adjoint embedding kernels stream them.
constexpr int kRowStoreCap = 192;  // neighbour slots per atom the store holds (sum of sel)

// The blocks whose rows the store holds.
__device__ __forceinline__ bool row_store_covers(const SysDesc &D, const float4 *rows_g, int nim) {
  return rows_g != nullptr && nim == 1 && D.S <= kRowStoreCap;
}

// One round of a row stream: the unread rows of earlier rounds move to the
// front (as in mix_compact_round), then up to RPT * blockDim rows [base,
// total) of the stored list are appended, RPT coalesced 16-byte loads per
// thread issued before any store.
template <int RPT>
__device__ __forceinline__ void mix_stream_round(const float4 *__restrict__ src, int base, int total, float4 *rowbuf,
                                                 int &rowstart, int &rowcount) {
  const int tid = threadIdx.x;
  if (rowstart > 0) {
    const int rem = rowcount - rowstart;  // < 128 <= blockDim
    float4 carry = make_float4(0.f, 0.f, 0.f, 0.f);
    if (tid < rem) carry = rowbuf[rowstart + tid];
    __syncthreads();
    if (tid < rem) rowbuf[tid] = carry;
    rowstart = 0;
    rowcount = rem;
  }
  const int n = min(RPT * (int)blockDim.x, total - base);
  float4 v[RPT];
#pragma unroll
  for (int k = 0; k < RPT; ++k) {
    const int i = tid + k * (int)blockDim.x;
    if (i < n) v[k] = src[base + i];
  }
#pragma unroll
  for (int k = 0; k < RPT; ++k) {
    const int i = tid + k * (int)blockDim.x;
    if (i < n) rowbuf[rowcount + i] = v[k];
  }
  rowcount += n;
  __syncthreads();
}

// Type-sorted positions with the frame-local user index, and the row store
// (rows.cu).
int launch_pos_sorted(const SysDesc &D, const float *pos, const int32_t *perm, float4 *posS, cudaStream_t st);
int launch_rows(const DevModel &M, const SysDesc &D, int ba, const float4 *posS, const float *box,
                const int32_t *nbrs, float4 *rows, int *rcnt, cudaStream_t st);

}  // namespace dpb

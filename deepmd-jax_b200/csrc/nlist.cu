// Typed neighbour list (cell binning + per-centre scan), sm_100a.
//
// Semantics (bit-exact target): the reference canonicalises coordinates as
// (coord % box) * (ref/box) * (1 - 5e-7) in float32 and sorts atoms by type
// (deepmd_jax/md_utils.py:364-373); jax_md's dense neighbour list keeps j != i
// with float32 d2 < cutoff^2 where d = mod(Ri - Rj + L/2, L) - L/2; get_nm
// (md_utils.py:431-459) then keeps per neighbour type the sel_j smallest
// indices in ascending order, type-local, padded with N, and flags overflow
// when more than sel_j exist.
//
// Layout: cells are binned per frame and each cell slot holds its atom's
// canonical position and index as one float4 (cell order), so a candidate is
// one coalesced 16-byte load.  A warp owns one centre atom, centres taken in
// cell order so that the warps of a block share their neighbourhood in L1.
// Cells are at least rc / 2 wide (at least rc where that would leave cells
// mostly empty).  Each lane takes one z-row of the 5 x 5 (3 x 3) rows around the
// centre, drops it if it lies outside the cutoff sphere and else cuts it to the
// sphere's chord; the rows' candidates are then walked as one flat sequence, 32
// per round with every lane busy.  Hits are appended per type into shared memory
// with ballots, sorted in registers, and the sorted prefix is written into the
// centre's own row.
//
// What bounds it: instruction issue (79 % of slots, the ALU pipe 69 % busy).
// With cells of rc, 98,304 atoms of liquid water at rc 6.3 A had 964 candidates in
// 36 rounds per centre: 505 us.  Cells of rc / 2 with the sphere cuts took it to
// 274 us, sorting in registers to 240 us, branch-free displacements to 217 us; 32
// frames of 1,536 atoms 474 -> 114 us.
#include "dpb_common.cuh"
#include <algorithm>
#include <climits>
#include <cmath>

namespace dpb {

struct NlGrid {
  int nc[3];
  int ncell;      // per frame
  int reach;      // cells on each side of the centre's that can hold neighbours
  int image_mode; // 1: some L < 2 rc, brute force over the frame's atoms
};

static NlGrid cell_grid(const float box[3], float rc, int reach) {
  NlGrid g;
  g.reach = reach;
  g.image_mode = 0;
  long long n = 1;
  for (int d = 0; d < 3; ++d) {
    g.nc[d] = std::max(1, std::min((int)floorf(box[d] * (float)reach / rc), 512));
    while (g.nc[d] > 1 && (double)box[d] * reach < (double)rc * g.nc[d]) --g.nc[d];
    // where cells beyond `reach` exist, cells wide enough that rounding brings no atom of theirs within rc
    while (g.nc[d] > 2 * reach + 1 && (double)box[d] * reach < ((double)rc + box[d] * 0x1p-20) * g.nc[d]) --g.nc[d];
    n *= g.nc[d];
    if (box[d] < 2.f * rc) g.image_mode = 1;
  }
  if (g.image_mode) {
    g.nc[0] = g.nc[1] = g.nc[2] = 1;
    n = 1;
  }
  g.ncell = (int)n;
  return g;
}

// Cells of rc / 2 where they hold an atom each on average, else of rc.
static NlGrid make_grid(const float box[3], float rc, int natoms) {
  const NlGrid fine = cell_grid(box, rc, 2);
  return fine.ncell <= natoms ? fine : cell_grid(box, rc, 1);
}

// A non-null gate makes every kernel of the build a no-op unless *gate != 0,
// so the rebuild can sit inside a captured MD step and run only when the
// drift test asks for it.
__global__ void nl_zero_kernel(int *__restrict__ a, int na, int *__restrict__ b, int nb,
                               const unsigned *__restrict__ gate) {
  if (gate && *gate == 0u) return;
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < na) a[i] = 0;
  if (i < nb) b[i] = 0;
}

// dbox (device, (F,3)) replaces L and scale = RB / L when the box changes on
// the device (NPT): the reference's canonicalize(coord, box) with the current
// box (md_utils.py:364-373).
__global__ void nl_canon_kernel(const float *__restrict__ pos, const int32_t *__restrict__ perm,
                                int N, int F, float3 L, float3 scale, float3 RB, int3 nc,
                                float *__restrict__ canon, int *__restrict__ atom_cell,
                                int *__restrict__ cell_count, const unsigned *__restrict__ gate,
                                const float *__restrict__ dbox) {
  if (gate && *gate == 0u) return;
  int g = blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= N * F) return;
  int f = g / N, k = g - f * N;
  if (dbox) {
    L = make_float3(dbox[f * 3], dbox[f * 3 + 1], dbox[f * 3 + 2]);
    scale = make_float3(__fdiv_rn(RB.x, L.x), __fdiv_rn(RB.y, L.y), __fdiv_rn(RB.z, L.z));
  }
  int src = perm ? perm[k] : k;
  const float *p = pos + ((size_t)f * N + src) * 3;
  const float shrink = 0.9999995f;  // float32(1 - 5e-7)
  float c0 = __fmul_rn(__fmul_rn(jmod(p[0], L.x), scale.x), shrink);
  float c1 = __fmul_rn(__fmul_rn(jmod(p[1], L.y), scale.y), shrink);
  float c2 = __fmul_rn(__fmul_rn(jmod(p[2], L.z), scale.z), shrink);
  canon[(size_t)g * 3 + 0] = c0;
  canon[(size_t)g * 3 + 1] = c1;
  canon[(size_t)g * 3 + 2] = c2;
  if (!cell_count) return;  // image mode
  // cell bins of the reference box (canonical coordinates live in [0, ref))
  int ix = min(max((int)(c0 / RB.x * nc.x), 0), nc.x - 1);
  int iy = min(max((int)(c1 / RB.y * nc.y), 0), nc.y - 1);
  int iz = min(max((int)(c2 / RB.z * nc.z), 0), nc.z - 1);
  int cell = (ix * nc.y + iy) * nc.z + iz;
  atom_cell[g] = cell;
  atomicAdd(&cell_count[f * (nc.x * nc.y * nc.z) + cell], 1);
}

// Exclusive scan of n ints with one block, 16 per thread and pass (four 16-byte
// loads in flight: 4 per thread took 14 us for the 29,791 cells of 98,304 atoms,
// one load latency and two barriers per 4,096 cells).
__global__ void __launch_bounds__(1024) nl_scan_kernel(const int *__restrict__ in, int *__restrict__ out, int n,
                                                      const unsigned *__restrict__ gate) {
  if (gate && *gate == 0u) return;
  __shared__ int part[32];
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  int run = 0;
  for (int base = 0; base < n; base += 16384) {
    const int i = base + 16 * t;
    int v[16], mine = 0;
    if (i + 16 <= n) {
#pragma unroll
      for (int k = 0; k < 16; k += 4) {
        const int4 q = *reinterpret_cast<const int4 *>(in + i + k);
        v[k] = q.x; v[k + 1] = q.y; v[k + 2] = q.z; v[k + 3] = q.w;
      }
    } else {
#pragma unroll
      for (int k = 0; k < 16; ++k) v[k] = i + k < n ? in[i + k] : 0;
    }
#pragma unroll
    for (int k = 0; k < 16; ++k) mine += v[k];
    int incl = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += u;
    }
    if (lane == 31) part[warp] = incl;
    __syncthreads();
    int w = part[lane];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= o) w += u;
    }
    const int before = __shfl_sync(0xffffffffu, w, warp ? warp - 1 : 0), total = __shfl_sync(0xffffffffu, w, 31);
    int e = run + (warp ? before : 0) + incl - mine;
#pragma unroll
    for (int k = 0; k < 16; ++k) {
      const int u = v[k];
      v[k] = e;
      e += u;
    }
    if (i + 16 <= n) {
#pragma unroll
      for (int k = 0; k < 16; k += 4)
        *reinterpret_cast<int4 *>(out + i + k) = make_int4(v[k], v[k + 1], v[k + 2], v[k + 3]);
    } else {
#pragma unroll
      for (int k = 0; k < 16; ++k)
        if (i + k < n) out[i + k] = v[k];
    }
    run += total;
    __syncthreads();
  }
  if (t == 0) out[n] = run;
}

__global__ void nl_scatter_kernel(const int *__restrict__ atom_cell, const int *__restrict__ cell_start,
                                  int *__restrict__ cursor, const float *__restrict__ canon,
                                  float4 *__restrict__ cell_pos, int N, int F, int ncell,
                                  const unsigned *__restrict__ gate) {
  if (gate && *gate == 0u) return;
  int g = blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= N * F) return;
  int f = g / N;
  int c = f * ncell + atom_cell[g];
  const int q = cell_start[c] + atomicAdd(&cursor[c], 1);
  cell_pos[q] = make_float4(canon[(size_t)g * 3], canon[(size_t)g * 3 + 1], canon[(size_t)g * 3 + 2],
                            __int_as_float(g - f * N));  // frame-local sorted index
}

struct NlParams {
  int N, F, ntypes, cap;
  int offs[kMaxTypes + 1];
  int sel[kMaxTypes];
  int col[kMaxTypes + 1];
  float3 L;      // reference box (canonical frame)
  float rc2;
  int3 nc;
  float3 h, inv_h;  // cell sizes
  float rcm2;    // squared cutoff with a margin, for the row cuts
  int reach, image_mode;
};

// Append the hits of one 32-candidate round into the per-type lists; the
// per-type counts are warp-uniform registers.  Hits past cap are dropped
// (that count is flagged as an overflow), in traversal order.
__device__ __forceinline__ void append_hits(bool hit, int t, int key, int ntypes, int cap, int (&cnt)[kMaxTypes],
                                            int *lists) {
  const unsigned lt = (1u << (threadIdx.x & 31)) - 1u;
#pragma unroll
  for (int tt = 0; tt < kMaxTypes; ++tt) {
    if (tt >= ntypes) break;
    const bool mine = hit && t == tt;
    const unsigned m = __ballot_sync(0xffffffffu, mine);
    if (mine) {
      const int p = cnt[tt] + __popc(m & lt);
      if (p < cap) lists[tt * cap + p] = key;
    }
    cnt[tt] += __popc(m);
  }
}

// Sorts up to 32 R distinct keys of a hit list ascending in registers (bitonic,
// element lane R + r: strides below R stay within a lane) and writes the first
// sel of them minus off.  Counting each key's smaller ones instead took about
// 650 instructions per centre (35 + 70 keys), this about 300.
template <int R>
__device__ __forceinline__ void sort_write(const int *__restrict__ L_, int nn, int sel, int off,
                                           int32_t *__restrict__ out) {
  const int lane = threadIdx.x & 31;
  int v[R];
#pragma unroll
  for (int r = 0; r < R; ++r) v[r] = lane * R + r < nn ? L_[lane * R + r] : INT_MAX;
#pragma unroll
  for (int k = 2; k <= 32 * R; k <<= 1)
#pragma unroll
    for (int j = k >> 1; j > 0; j >>= 1) {
      if (j >= R) {  // partner element in another lane
        const bool keep_min = ((lane * R & j) == 0) == ((lane * R & k) == 0);
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const int o = __shfl_xor_sync(0xffffffffu, v[r], j / R);
          v[r] = keep_min ? min(v[r], o) : max(v[r], o);
        }
      } else {
#pragma unroll
        for (int r = 0; r < R; ++r)
          if ((r & j) == 0) {
            const bool up = ((lane * R + r) & k) == 0;
            const int lo = min(v[r], v[r | j]), hi = max(v[r], v[r | j]);
            v[r] = up ? lo : hi;
            v[r | j] = up ? hi : lo;
          }
      }
    }
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int e = lane * R + r;
    if (e < nn && e < sel) out[e] = v[r] - off;
  }
}

// jax_md.space.periodic displacement of one axis, mod(ci - cj + L/2, L) - L/2 in
// float32.  Canonical coordinates lie in [0, L), so the argument lies in (-L/2,
// 3L/2) and its mod is one exact or correctly rounded add (jmod in branch-free
// form).
__device__ __forceinline__ float canon_disp(float ci, float cj, float L, float h) {
  const float t = __fadd_rn(__fsub_rn(ci, cj), h);
  const float w = t < 0.f ? L : t >= L ? -L : 0.f;
  return __fsub_rn(__fadd_rn(t, w), h);
}

__device__ __forceinline__ bool pair_hit(float3 ci, float3 cj, float3 L, float rc2) {
  const float dx = canon_disp(ci.x, cj.x, L.x, 0.5f * L.x), dy = canon_disp(ci.y, cj.y, L.y, 0.5f * L.y),
              dz = canon_disp(ci.z, cj.z, L.z, 0.5f * L.z);
  const float d2 = __fadd_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)), __fmul_rn(dz, dz));
  return d2 < rc2;
}

// First offset and number of the cells to visit along an axis of nc cells: every
// cell once where fewer than 2 reach + 1 exist.
__device__ __forceinline__ int2 nl_span(int nc, int reach) {
  return nc >= 2 * reach + 1 ? make_int2(-reach, 2 * reach + 1) : make_int2(-((nc - 1) / 2), nc);
}

// Distance (in cells) from a point at fraction fr of its cell to the cells at
// offset o; 0 where the axis has so few cells that o stands for two images.
__device__ __forceinline__ float nl_gap(int o, float fr, int nc, int reach) {
  const float d = o > 0 ? (float)o - fr : o < 0 ? fr - (float)(o + 1) : 0.f;
  return nc >= 2 * reach + 1 ? fmaxf(d, 0.f) : 0.f;
}

// 48 registers: 40 resident warps per SM at every launch shape (128-512
// threads), with nothing spilled.
__global__ void __maxnreg__(48) nl_search_kernel(NlParams P, const float *__restrict__ canon,
                                                 const int *__restrict__ cell_start,
                                                 const float4 *__restrict__ cell_pos,
                                                 int32_t *__restrict__ nbrs,
                                                 int32_t *__restrict__ counts,
                                                 uint32_t *__restrict__ status,
                                                 const unsigned *__restrict__ gate) {
  if (gate && *gate == 0u) return;
  extern __shared__ __align__(16) int smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int wpb = blockDim.x >> 5;
  int4 *rows = reinterpret_cast<int4 *>(smem) + warp * 32;  // the rows' (first candidate, range 1, its length, range 2)
  int *lists = smem + wpb * 128 + warp * P.ntypes * P.cap;
  const int gc = blockIdx.x * wpb + warp;  // position in cell order (image mode: in sorted order)
  if (gc >= P.N * P.F) return;
  const int f = gc / P.N;
  const float *cf = canon + (size_t)f * P.N * 3;
  int i = gc - f * P.N;  // frame-local sorted index of the centre
  float3 ci;
  int cnt[kMaxTypes] = {0, 0, 0, 0};

  if (!P.image_mode) {
    const float4 c4 = cell_pos[gc];
    i = __float_as_int(c4.w);
    ci = make_float3(c4.x, c4.y, c4.z);
    const int ncell = P.nc.x * P.nc.y * P.nc.z, nz = P.nc.z;
    const int *cs = cell_start + f * ncell;
    const int ix = min(max((int)(ci.x / P.L.x * P.nc.x), 0), P.nc.x - 1);
    const int iy = min(max((int)(ci.y / P.L.y * P.nc.y), 0), P.nc.y - 1);
    const int iz = min(max((int)(ci.z / P.L.z * P.nc.z), 0), P.nc.z - 1);
    const int2 sx = nl_span(P.nc.x, P.reach), sy = nl_span(P.nc.y, P.reach), sz = nl_span(nz, P.reach);
    // ---- this lane's z-row: one or two ranges of cell order
    int b1 = 0, n1 = 0, b2 = 0, n2 = 0;
    if (lane < sx.y * sy.y) {
      const int rx = lane / sy.y, ox = sx.x + rx, oy = sy.x + lane - rx * sy.y;
      const float gx = nl_gap(ox, ci.x * P.inv_h.x - (float)ix, P.nc.x, P.reach) * P.h.x;
      const float gy = nl_gap(oy, ci.y * P.inv_h.y - (float)iy, P.nc.y, P.reach) * P.h.y;
      const float rem = P.rcm2 - gx * gx - gy * gy;
      if (rem > 0.f) {
        int z0 = iz + sz.x, z1 = z0 + sz.y - 1;
        if (nz >= 2 * P.reach + 1) {  // the chord of the sphere
          const float zc = ci.z * P.inv_h.z, zr = sqrtf(rem) * P.inv_h.z;
          z0 = max(z0, (int)floorf(zc - zr));
          z1 = min(z1, (int)floorf(zc + zr));
        }
        // ix + ox lies in [-nc, 2 nc), so one conditional add or subtract wraps it
        int cx = ix + ox, cy = iy + oy;
        cx += cx < 0 ? P.nc.x : 0;
        cx -= cx >= P.nc.x ? P.nc.x : 0;
        cy += cy < 0 ? P.nc.y : 0;
        cy -= cy >= P.nc.y ? P.nc.y : 0;
        const int *row = cs + (cx * P.nc.y + cy) * nz;
        int a0 = z0, a1 = z1;
        if (z0 < 0) {
          a0 = z0 + nz;
          a1 = nz - 1;
          b2 = row[0];
          n2 = row[z1 + 1] - b2;
        } else if (z1 >= nz) {
          a1 = nz - 1;
          b2 = row[0];
          n2 = row[z1 - nz + 1] - b2;
        }
        b1 = row[a0];
        n1 = row[a1 + 1] - b1;
      }
    }
    // ---- the rows with candidates, in order, as one flat sequence
    const int n = n1 + n2;
    int incl = n;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += u;
    }
    const int total = __shfl_sync(0xffffffffu, incl, 31), start = incl - n;
    const unsigned live = __ballot_sync(0xffffffffu, n > 0), lt = (1u << lane) - 1u, le = lt | (1u << lane);
    if (n > 0) rows[__popc(live & lt)] = make_int4(start, b1, n1, b2);
    __syncwarp();
    int before = 0;  // rows that start before this round
    for (int base = 0; base < total; base += 32) {
      // bit l: a row starts at candidate base + l
      const unsigned off = (unsigned)(start - base);
      const unsigned starts = __reduce_or_sync(0xffffffffu, n > 0 && off < 32u ? 1u << off : 0u);
      const int p = base + lane;
      bool hit = false;
      int j = 0, t = 0;
      if (p < total) {
        const int4 r = rows[before + __popc(starts & le) - 1];
        const int k = p - r.x;
        const float4 v = cell_pos[k < r.z ? r.y + k : r.w + k - r.z];
        j = __float_as_int(v.w);
        hit = (j != i) && pair_hit(ci, make_float3(v.x, v.y, v.z), P.L, P.rc2);
        t = type_of(j, P.offs, P.ntypes);
      }
      before += __popc(starts);
      append_hits(hit, t, j, P.ntypes, P.cap, cnt, lists);
    }
  } else {
    // Some L < 2 rc: j is listed once if any periodic image lies within rc.
    // For j != i that is the nearest image (|d + m L| >= |d| per axis for every m,
    // in floating point too: d + L >= L / 2 >= |d| before rounding, which is
    // monotonic); for j == i the nearest image that is not the atom itself.
    ci = make_float3(cf[i * 3], cf[i * 3 + 1], cf[i * 3 + 2]);
    const float ls = fminf(P.L.x, fminf(P.L.y, P.L.z));
    const bool self = ls * ls < P.rc2;
    for (int base = 0; base < P.N; base += 32) {
      const int j = base + lane;
      bool hit = false;
      int t = 0;
      if (j < P.N) {
        const float x = shift_ortho(cf[j * 3] - ci.x, P.L.x), y = shift_ortho(cf[j * 3 + 1] - ci.y, P.L.y),
                    z = shift_ortho(cf[j * 3 + 2] - ci.z, P.L.z);
        hit = j == i ? self : x * x + y * y + z * z < P.rc2;
        t = type_of(j, P.offs, P.ntypes);
      }
      append_hits(hit, t, j, P.ntypes, P.cap, cnt, lists);
    }
  }
  const int g = f * P.N + i;
  // sort each type's hits and write the sel_t smallest
  const int S = P.col[P.ntypes];
  int32_t *out = nbrs + (size_t)g * S;
  bool ovf = false;
#pragma unroll 1
  for (int t = 0; t < P.ntypes; ++t) {
    const int n = t == 0 ? cnt[0] : t == 1 ? cnt[1] : t == 2 ? cnt[2] : cnt[3];
    if (counts && lane == 0) counts[(size_t)g * P.ntypes + t] = n;
    ovf |= (n > P.sel[t]) || (n > P.cap);
    const int nn = min(n, P.cap);
    const int *L_ = lists + t * P.cap;
    __syncwarp();
    int32_t *o = out + P.col[t];
    const int sel = P.sel[t], off = P.offs[t];
    if (nn <= 32) sort_write<1>(L_, nn, sel, off, o);
    else if (nn <= 64) sort_write<2>(L_, nn, sel, off, o);
    else if (nn <= 128) sort_write<4>(L_, nn, sel, off, o);
    else  // long lists (large sel): one key per lane at a time, few registers
      for (int e = lane; e < nn; e += 32) {
        const int key = L_[e];
        int rank = 0;
        for (int e2 = 0; e2 < nn; ++e2) rank += (L_[e2] < key);
        if (rank < sel) o[rank] = key - off;
      }
    for (int e = nn + lane; e < sel; e += 32) o[e] = P.N;
  }
  if (ovf && lane == 0) atomicOr(status, DPB_ST_NLIST_OVERFLOW);
}

}  // namespace dpb

using namespace dpb;

static size_t align_up(size_t x) { return (x + 255) & ~(size_t)255; }

static size_t nlist_bytes(size_t NF, size_t C) {
  return align_up(C * 4) * 2 + align_up((C + 1) * 4) + align_up(NF * 4) + align_up(NF * 16) + align_up(NF * 12);
}

// Enough for both cell sizes of make_grid, and monotonic in rc: a caller may
// size the workspace at a slightly smaller cutoff than it builds with.
extern "C" int dpb_nlist_workspace_bytes(int natoms, int nframes, const float box[3], float rc,
                                         size_t *bytes) {
  if (!bytes || natoms <= 0 || nframes <= 0 || !box || rc <= 0) return DPB_ERR_INVALID_ARG;
  const int ncell = std::max(cell_grid(box, rc, 1).ncell, std::min(cell_grid(box, rc, 2).ncell, natoms));
  *bytes = nlist_bytes((size_t)natoms * nframes, (size_t)ncell * nframes);
  return DPB_OK;
}

namespace dpb {
int nlist_build_impl(const float *pos, const int32_t *perm, int natoms, int nframes, int ntypes,
                     const int *type_count, const int *sel, const float box[3], const float *ref_box, float rc,
                     int32_t *nbrs, float *ref_pos, int32_t *counts, uint32_t *status, void *workspace,
                     size_t ws_bytes, const unsigned *gate, cudaStream_t stream, const float *dbox,
                     int nl_warps) {
  if (!pos || natoms <= 0 || nframes <= 0 || ntypes < 1 || ntypes > kMaxTypes || !type_count || !sel ||
      !box || !nbrs || !status || rc <= 0)
    return DPB_ERR_INVALID_ARG;
  if (natoms >= (1 << 24)) return DPB_ERR_UNSUPPORTED;
  float rb[3] = {box[0], box[1], box[2]};
  if (ref_box) { rb[0] = ref_box[0]; rb[1] = ref_box[1]; rb[2] = ref_box[2]; }
  // jax_md receives rcut * max(ref/box) as float32 and squares it in float32
  float smax = std::max(rb[0] / box[0], std::max(rb[1] / box[1], rb[2] / box[2]));
  float rc_eff = rc * smax;
  NlGrid g = make_grid(rb, rc_eff, natoms);
  if (g.image_mode)
    for (int d = 0; d < 3; ++d)  // more than 4 images of an axis within reach
      if ((int)floorf(rc_eff / rb[d] + 0.5f) > 4) return DPB_ERR_UNSUPPORTED;
  const size_t NF = (size_t)natoms * nframes;
  if (ws_bytes < nlist_bytes(NF, (size_t)g.ncell * nframes)) g = cell_grid(rb, rc_eff, 1);
  if (!workspace || ws_bytes < nlist_bytes(NF, (size_t)g.ncell * nframes)) return DPB_ERR_WORKSPACE;
  NlParams P;
  P.N = natoms; P.F = nframes; P.ntypes = ntypes;
  int smax_sel = 0, off = 0, col = 0;
  for (int t = 0; t < ntypes; ++t) {
    if (type_count[t] < 0 || sel[t] < 0) return DPB_ERR_INVALID_ARG;
    P.offs[t] = off; off += type_count[t];
    P.sel[t] = sel[t]; P.col[t] = col; col += sel[t];
    smax_sel = std::max(smax_sel, sel[t]);
  }
  if (off != natoms) return DPB_ERR_INVALID_ARG;
  for (int t = ntypes; t <= kMaxTypes; ++t) P.offs[t] = natoms;
  P.col[ntypes] = col;
  // hit buffer per type: the sorted prefix is exact whenever a type's count
  // fits (counts above cap only occur with overflow already flagged)
  int cap = 256;
  while (cap < smax_sel + 1) cap <<= 1;
  if (cap > 1024) return DPB_ERR_UNSUPPORTED;
  P.cap = cap;
  P.L = make_float3(rb[0], rb[1], rb[2]);
  P.rc2 = rc_eff * rc_eff;
  P.nc = make_int3(g.nc[0], g.nc[1], g.nc[2]);
  P.image_mode = g.image_mode;
  P.reach = g.reach;
  P.h = make_float3(rb[0] / g.nc[0], rb[1] / g.nc[1], rb[2] / g.nc[2]);
  P.inv_h = make_float3(1.f / P.h.x, 1.f / P.h.y, 1.f / P.h.z);
  // above the rounding of bins, gaps (3 x 2^-24 L) and displacements (2^-21 L), also in a box so long
  // that a float's step in it is no longer small
  const float rcm = rc_eff * 1.0001f + 1e-3f + 0x1p-20f * std::max(rb[0], std::max(rb[1], rb[2]));
  P.rcm2 = rcm * rcm;

  const size_t C = (size_t)g.ncell * nframes;
  char *w = (char *)workspace;
  int *cell_count = (int *)w; w += align_up(C * 4);
  int *cursor = (int *)w; w += align_up(C * 4);
  int *cell_start = (int *)w; w += align_up((C + 1) * 4);
  int *atom_cell = (int *)w; w += align_up(NF * 4);
  float4 *cell_pos = (float4 *)w; w += align_up(NF * 16);
  float *canon = ref_pos ? ref_pos : (float *)w;

  float3 L = make_float3(box[0], box[1], box[2]);
  float3 scale = make_float3(rb[0] / box[0], rb[1] / box[1], rb[2] / box[2]);
  int nb = (int)((NF + 255) / 256);
  if (!g.image_mode) {
    nl_zero_kernel<<<(int)((C + 255) / 256), 256, 0, stream>>>(cell_count, (int)C, cursor, (int)C, gate);
    count_launch();
  }
  nl_canon_kernel<<<nb, 256, 0, stream>>>(pos, perm, natoms, nframes, L, scale, P.L, P.nc, canon, atom_cell,
                                          g.image_mode ? nullptr : cell_count, gate, dbox);
  if (!g.image_mode) {
    nl_scan_kernel<<<1, 1024, 0, stream>>>(cell_count, cell_start, (int)C, gate);
    nl_scatter_kernel<<<nb, 256, 0, stream>>>(atom_cell, cell_start, cursor, canon, cell_pos, natoms, nframes,
                                              g.ncell, gate);
    count_launch(2);
  }
  if (nl_warps != 4 && nl_warps != 8 && nl_warps != 16) return DPB_ERR_INVALID_ARG;
  const int wpb = nl_warps, threads = 32 * wpb;  // centres (warps) per block
  size_t smem = (size_t)wpb * (512 + (size_t)ntypes * cap * 4);
  if (smem > 200 * 1024) return DPB_ERR_UNSUPPORTED;  // hit lists of this many warps do not fit
  if (smem > 48 * 1024) {
    DPB_CUDA_TRY(cudaFuncSetAttribute(nl_search_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  }
  nl_search_kernel<<<(int)((NF + wpb - 1) / wpb), threads, smem, stream>>>(P, canon, cell_start, cell_pos, nbrs,
                                                                           counts, status, gate);
  count_launch(2);
  DPB_LAUNCH_CHECK();
  return DPB_OK;
}
}  // namespace dpb

extern "C" int dpb_nlist_build(const float *pos, const int32_t *perm, int natoms, int nframes, int ntypes,
                               const int *type_count, const int *sel, const float box[3],
                               const float *ref_box, float rc, int32_t *nbrs, float *ref_pos,
                               int32_t *counts, uint32_t *status, void *workspace, size_t ws_bytes,
                               void *stream) {
  return dpb::nlist_build_impl(pos, perm, natoms, nframes, ntypes, type_count, sel, box, ref_box, rc, nbrs,
                               ref_pos, counts, status, workspace, ws_bytes, nullptr, (cudaStream_t)stream,
                               nullptr, 8);
}

// ---------------------------------------------------------------- packed batches
namespace dpb {
// Where the frames of one request land in a packed batch: frame f's type-t
// atoms are packed rows row0[t] + f * stride[t] + m (m < count of type t), and
// its type-t atom m is type-local index base0[t] + f * stride[t] + m of the
// packed type block.
struct PackMap {
  int ntypes, S, Ns, nframes, Np;
  int soffs[kMaxTypes + 1];
  int col[kMaxTypes + 1];
  int row0[kMaxTypes], base0[kMaxTypes], stride[kMaxTypes];
};

__global__ void nl_pack_kernel(const int32_t *__restrict__ src, PackMap m, int32_t *__restrict__ dst) {
  const size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  const size_t per_frame = (size_t)m.Ns * m.S;
  if (e >= per_frame * m.nframes) return;
  const int f = (int)(e / per_frame);
  const size_t rc = e - (size_t)f * per_frame;
  const int r = (int)(rc / m.S), c = (int)(rc - (size_t)r * m.S);
  int i = 0, j = 0;
  while (i + 1 < m.ntypes && r >= m.soffs[i + 1]) ++i;
  while (j + 1 < m.ntypes && c >= m.col[j + 1]) ++j;
  const int v = src[e] & DPB_NBR_INDEX_MASK;
  const int cnt_j = m.soffs[j + 1] - m.soffs[j];
  const int out = v < cnt_j ? m.base0[j] + f * m.stride[j] + v : m.Np;
  const size_t row = (size_t)m.row0[i] + (size_t)f * m.stride[i] + (r - m.soffs[i]);
  dst[row * m.S + c] = out;
}
}  // namespace dpb

extern "C" int dpb_nlist_pack(const int32_t *src, int natoms, int nframes, int ntypes, const int *type_count,
                              const int *sel, const int *row0, const int *base0, const int *stride,
                              int packed_natoms, int32_t *dst, void *stream) {
  if (!src || !dst || !type_count || !sel || !row0 || !base0 || !stride || natoms <= 0 || nframes <= 0 ||
      ntypes < 1 || ntypes > dpb::kMaxTypes || packed_natoms <= 0)
    return DPB_ERR_INVALID_ARG;
  dpb::PackMap m;
  m.ntypes = ntypes; m.Ns = natoms; m.nframes = nframes; m.Np = packed_natoms;
  int off = 0, col = 0;
  for (int t = 0; t < ntypes; ++t) {
    if (type_count[t] < 0 || sel[t] < 0 || stride[t] < type_count[t]) return DPB_ERR_INVALID_ARG;
    m.soffs[t] = off; off += type_count[t];
    m.col[t] = col; col += sel[t];
    m.row0[t] = row0[t]; m.base0[t] = base0[t]; m.stride[t] = stride[t];
    if (row0[t] < 0 || base0[t] < 0 || (long long)row0[t] + (long long)stride[t] * nframes > packed_natoms)
      return DPB_ERR_INVALID_ARG;
  }
  if (off != natoms) return DPB_ERR_INVALID_ARG;
  m.soffs[ntypes] = off; m.col[ntypes] = col; m.S = col;
  const size_t n = (size_t)natoms * col * nframes;
  if (n == 0) return DPB_OK;
  dpb::nl_pack_kernel<<<(unsigned)((n + 255) / 256), 256, 0, (cudaStream_t)stream>>>(src, m, dst);
  dpb::count_launch();
  DPB_LAUNCH_CHECK();
  return DPB_OK;
}

// FP32 fitting GEMMs on the tensor cores: C = A B with A (atoms x K) split on
// the fly into FP16 hi + lo parts and the weights into three FP16 parts (exact
// to 33 bits), four products lo.hi, hi.lo2, hi.lo, hi.hi per K step, smallest
// first.  The tensor core truncates its FP32 accumulator at every K = 16 step
// (about half a unit in the last place lost each time, measured), so every 32
// of K the partial sum leaves TMEM and is added in registers with rounding to
// nearest: against float64 the sums are closer than the 1,600-term
// multiply-add chains that they replace.
//
// Operand scales are powers of two: the weights' per layer, hidden activations'
// from bounds known at model creation, the descriptor's per atom from its largest
// entry (gmax, written with G), the gates' per atom and 32 columns from their largest
// entry (a bound down all layers left wide deep nets 11 bits: force error 3.2e-6 of
// the rms force at 1024^4, 5e-7 now), all divided out of the sum exactly.
#include <type_traits>

#include "internal.cuh"
#include "tc.cuh"

namespace dpb {

constexpr int kGemmTile = 128;                        // rows of a stored weight tile
constexpr int kGemmChunk = 3 * 4 * kGemmTile * 16;    // bytes of one stored weight chunk: hi, lo, lo2

// Stored weight chunks of one matrix: B[n][k] = w[n sn + k sk], n < N, k < K, as
// [n tile][k chunk][part][k8][row][8] FP16 of w times scale, zero padded.
__global__ void k_gemm_tiles(const float *__restrict__ w, int N, int K, int sn, int sk, float scale,
                             __half *__restrict__ out, int total) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;  // (tile, chunk, k8, row, e)
  if (i >= total) return;
  const int e = i & 7, r = (i >> 3) & 127, k8 = (i >> 10) & 3, tc_ = i >> 12;
  const int nc = (K + kGemmK - 1) / kGemmK, t = tc_ / nc, c = tc_ - t * nc;
  const int n = t * kGemmTile + r, k = c * kGemmK + 8 * k8 + e;
  const float v = (n < N && k < K) ? w[(size_t)n * sn + (size_t)k * sk] * scale : 0.f;
  const __half h = __float2half_rn(v);
  const float r1 = v - __half2float(h);  // exact
  const __half l = __float2half_rn(r1);
  __half *o = out + ((size_t)tc_ * 3 * 4 + k8) * 1024 + r * 8 + e;
  o[0] = h;
  o[4 * 1024] = l;
  o[8 * 1024] = __float2half_rn(r1 - __half2float(l));
}

size_t gemm_tiles_halves(int N, int K) {
  return (size_t)((N + kGemmTile - 1) / kGemmTile) * ((K + kGemmK - 1) / kGemmK) * (kGemmChunk / 2);
}

int launch_gemm_tiles(const float *w, int N, int K, int sn, int sk, float scale, __half *out) {
  const int total = (int)(gemm_tiles_halves(N, K) / 3);
  k_gemm_tiles<<<(total + 255) / 256, 256>>>(w, N, K, sn, sk, scale, out, total);
  DPB_LAUNCH_CHECK();
  return DPB_OK;
}

// Power of two that brings x into [2^13, 2^14) (exponent within +-60); 1 for 0
// and non-finite x.
__device__ __forceinline__ float row_scale(float x) {
  if (!(x > 0.f) || !(x < INFINITY)) return 1.f;
  int e;
  frexpf(x, &e);
  return ldexpf(1.f, max(-60, min(60, 14 - e)));
}

// Persistent CTAs (one per SM) over tiles of 128 rows (atoms of one centre type)
// x NW output columns, warp-specialised, K in chunks of 32 through a ring of
// three stages (A, weights and a TMEM accumulator each).  Layer 0 (TILED false):
//   warps 0-7   add each chunk's sum from TMEM to their registers (two threads
//               per row, half the columns each) and run the epilogue, while
//   warps 8-15  load A in FP32, split it and store the operand,
//   warp 16     issues the MMAs, and
//   warp 17     the bulk copies of the weights
// already work on the next tile.  Every other GEMM (TILED) finds A split and tiled
// by the epilogue before it (gemm_operand_at), so that A too comes by bulk copies
// and warps 8-15 are a second group of adders that takes every other tile: one
// group's epilogue overlaps the other's sums.
//
// What bounds it: the chain of an epilogue (128 x NW values through shared memory,
// tanh, 64 to 192 KB written), and per chunk the single threads' waits and issues
// (about 850 clocks, against the 520 of the MMAs).  98,304 atoms, all six GEMMs:
// 1,880 us with every A split by the warps of the tile that needs it (13 times for
// dE/dG), one group of adders, a division per row for the epilogue's addresses and
// 8-way bank conflicts in A's loads; 1,330 us without (layer 0 622 -> 567); the
// gates' scales per row and chunk cost 27 us of it.
constexpr int kGemmStages = 3;
constexpr int kGemmThreads = 18 * 32;

template <int NW, bool TILED>
struct GemmCfg {
  // A: bytes between 8-wide K groups (split here, 8-byte stores of a half warp fall
  // into different banks), and of a stage's hi and lo parts
  static constexpr int ALBO = TILED ? 2048 : 2048 + 32, AB = 2 * 4 * ALBO;
  static constexpr int BB = 3 * 4 * NW * 16, STAGE = AB + BB;
  static constexpr int ZS = NW + 4;  // row stride of the staged result (floats)
  static constexpr int SMEM = kGemmStages * STAGE + 128 * ZS * 4;
  static constexpr int TM = NW == 128 ? 512 : 4 * NW;  // TMEM columns (a power of two >= 3 NW)
};

// Bounded wait that also gives up once another role gave up.
__device__ __forceinline__ bool gemm_wait(uint64_t *bar, uint32_t parity, volatile int *abort) {
  const uint32_t a = tc::smem_u32(bar);
  for (int it = 0; it < tc::kWaitLimit; ++it) {
    if (tc::mbar_test(a, parity)) return true;
    if ((it & 31) == 31 && *abort) return false;
  }
  *abort = 1;
  return false;
}

struct GemmTilePos {
  int ti, mt, m0, n0, nv;
};
template <int NW>
__device__ __forceinline__ GemmTilePos gemm_tile(const GemmArgs &g, int tile) {
  const int ntn = (g.N + NW - 1) / NW, mt = tile / ntn;
  GemmTilePos p;
  p.mt = mt;
  p.n0 = (tile - mt * ntn) * NW;
  p.nv = min(NW, g.N - p.n0);
  p.ti = 0;
#pragma unroll
  for (int t = 1; t < kMaxTypes; ++t)
    if (t < g.ntypes && mt >= g.mt0[t]) p.ti = t;
  p.m0 = (mt - g.mt0[p.ti]) * 128;
  return p;
}

// Four consecutive columns, or one, of the next GEMM's operand, split as the
// loading warps split it.
__device__ __forceinline__ __half *gemm_tile_at(const Epi &ep, int mt, int lr, int n) {
  return ep.tile + gemm_operand_at((ep.ld + kGemmK - 1) / kGemmK, mt, lr, n);
}
__device__ __forceinline__ void gemm_tile_store4(const Epi &ep, int mt, int lr, int n, float4 v, float scale) {
  __half *o = gemm_tile_at(ep, mt, lr, n);
  const tc::f2 sc = tc::pk1(scale);
  uint2 h, l;
  tc::split_pair(tc::mul2(tc::pk(v.x, v.y), sc), h.x, l.x);
  tc::split_pair(tc::mul2(tc::pk(v.z, v.w), sc), h.y, l.y);
  *reinterpret_cast<uint2 *>(o) = h;
  *reinterpret_cast<uint2 *>(o + kGemmPart) = l;
}
__device__ __forceinline__ void gemm_tile_store1(const Epi &ep, int mt, int lr, int n, float v, float scale) {
  __half *o = gemm_tile_at(ep, mt, lr, n);
  const float x = v * scale;
  const __half h = __float2half_rn(x);
  o[0] = h;
  o[kGemmPart] = __float2half_rn(x - __half2float(h));
}

// One column of an epilogue: x the GEMM's value, a the residual or adjoint
// addend (hprev, gmat or gvec), t the tanh value of the layer below.
template <int MODE>
__device__ __forceinline__ void gemm_epi1(float x, float bias, float dt, float a, float t, float &o1, float &o2) {
  if constexpr (MODE == EPI_STORE) {
    o1 = x;
  } else if constexpr (MODE == EPI_TANH) {
    o1 = o2 = tanhf(x + bias);
  } else if constexpr (MODE == EPI_TANH_RES) {
    o1 = tanhf(x + bias);
    o2 = o1 * dt + a;
  } else if constexpr (MODE == EPI_GRAD_RES) {
    o2 = x + a;
    o1 = o2 * dt * (1.f - t * t);
  } else {
    o1 = (x + a) * (1.f - t * t);
  }
}

// Epilogue of one tile by 8 warps: a warp takes 16 rows, RB at a time with all of
// their loads issued before any is used, lanes over column quads (single
// columns where the row length is no multiple of 4).
template <int NW, int MODE>
__device__ __forceinline__ void gemm_epilogue(const GemmType &gt, const GemmTilePos &p, const float *zs, float bad) {
  constexpr int ZS = GemmCfg<NW, true>::ZS, LQ = NW / 4, RPW = 32 / LQ;  // lanes per row, rows per warp pass
  constexpr int RM = MODE == EPI_GRAD || MODE == EPI_GRAD_RES ? 4 : 8, RB = 16 / RPW < RM ? 16 / RPW : RM;
  constexpr bool TANH = MODE == EPI_TANH || MODE == EPI_TANH_RES, GRAD = MODE == EPI_GRAD || MODE == EPI_GRAD_RES;
  const int warp = (threadIdx.x >> 5) & 7, lane = threadIdx.x & 31;
  const Epi &ep = gt.ep;
  const int n16 = (ep.ld + 15) / 16 * 16;  // the next GEMM reads whole K = 16 steps
  const int nc = (ep.ld + kGemmK - 1) / kGemmK;
  if ((ep.ld & 3) != 0) {
    for (int lr = warp; lr < 128 && p.m0 + lr < gt.Mrows; lr += 8) {
      const size_t at = gt.rm.atom(p.m0 + lr) * (size_t)ep.ld + p.n0;
      for (int j = lane; j - lane < NW && p.n0 + j - lane < n16; j += 32) {  // a warp takes 32 columns, one scale
        const int n = p.n0 + j;
        float o1 = 0.f, o2 = 0.f;
        if (j < p.nv) {
          const float *am = MODE == EPI_TANH_RES ? ep.hprev : ep.gmat;
          const float a = GRAD && ep.gvec ? ep.gvec[n] : (MODE == EPI_TANH_RES || GRAD) && am ? am[at + j] : 0.f;
          gemm_epi1<MODE>(zs[lr * ZS + j] + bad, TANH ? ep.bias[n] : 0.f,
                          MODE == EPI_TANH_RES || MODE == EPI_GRAD_RES ? ep.dt[n] : 1.f, a, GRAD ? ep.tin[at + j] : 0.f,
                          o1, o2);
          if (ep.out1) ep.out1[at + j] = o1;
          if (MODE != EPI_STORE && MODE != EPI_GRAD && ep.out2) ep.out2[at + j] = o2;
        }
        if (MODE == EPI_STORE || !ep.tile) continue;
        float sc = ep.tscale;
        if (GRAD) {
          float m = fabsf(o1);
#pragma unroll
          for (int o = 1; o < 32; o <<= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
          const int k = gate_exp(m);
          sc = pow2i(k);
          if (lane == 0) ep.texp[gemm_exp_at(nc, p.mt, lr, n / kGemmK)] = (int8_t)k;
        }
        if (n < n16) gemm_tile_store1(ep, p.mt, lr, n, GRAD ? o1 : o2, sc);
      }
    }
    return;
  }
  const int j = 4 * (lane % LQ), rl = lane / LQ;
  const bool on = j < p.nv, pad = !on && ep.tile && p.n0 + j < n16;
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
  auto ld4 = [&](const float *q) { return on ? *reinterpret_cast<const float4 *>(q) : zero; };
  const float4 bias = TANH ? ld4(ep.bias + p.n0 + j) : zero;
  const float4 dt = MODE == EPI_TANH_RES || MODE == EPI_GRAD_RES ? ld4(ep.dt + p.n0 + j) : zero;
  const float4 gv = GRAD && ep.gvec ? ld4(ep.gvec + p.n0 + j) : zero;
  const float *am = MODE == EPI_TANH_RES ? ep.hprev : GRAD && !ep.gvec ? ep.gmat : nullptr;
  // each lane's row of the warp's 16 (a division per row and warp took half of the
  // kernel's instructions)
  const int nrow = min(max(gt.Mrows - p.m0 - 16 * warp, 0), 16);
  const size_t at_l = (lane & 15) < nrow ? gt.rm.atom(p.m0 + 16 * warp + (lane & 15)) * (size_t)ep.ld + p.n0 : 0;
#pragma unroll 1
  for (int q = 0; q < 16; q += RB * RPW) {
    float4 a[RB], t[RB];
#pragma unroll
    for (int b = 0; b < RB; ++b) {
      const int r = q + b * RPW + rl;
      const size_t at = __shfl_sync(0xffffffffu, at_l, r) + j;
      a[b] = gv;
      t[b] = zero;
      if (on && r < nrow) {
        if ((MODE == EPI_TANH_RES || GRAD) && am) a[b] = *reinterpret_cast<const float4 *>(am + at);
        if (GRAD) t[b] = *reinterpret_cast<const float4 *>(ep.tin + at);
      }
    }
#pragma unroll
    for (int b = 0; b < RB; ++b) {
      const int r = q + b * RPW + rl, lr = 16 * warp + r;
      const size_t at = __shfl_sync(0xffffffffu, at_l, r) + j;
      float4 o1 = zero, o2 = zero;
      if (on && r < nrow) {
        const float4 x = *reinterpret_cast<const float4 *>(zs + lr * ZS + j);
        gemm_epi1<MODE>(x.x + bad, bias.x, dt.x, a[b].x, t[b].x, o1.x, o2.x);
        gemm_epi1<MODE>(x.y + bad, bias.y, dt.y, a[b].y, t[b].y, o1.y, o2.y);
        gemm_epi1<MODE>(x.z + bad, bias.z, dt.z, a[b].z, t[b].z, o1.z, o2.z);
        gemm_epi1<MODE>(x.w + bad, bias.w, dt.w, a[b].w, t[b].w, o1.w, o2.w);
        if (ep.out1) *reinterpret_cast<float4 *>(ep.out1 + at) = o1;
        if (MODE != EPI_STORE && MODE != EPI_GRAD && ep.out2) *reinterpret_cast<float4 *>(ep.out2 + at) = o2;
      }
      float sc = ep.tscale;
      if (GRAD) {  // 8 lanes hold a row's 32 columns
        float m = fmaxf(fmaxf(fabsf(o1.x), fabsf(o1.y)), fmaxf(fabsf(o1.z), fabsf(o1.w)));
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
        const int k = gate_exp(m);
        sc = pow2i(k);
        if ((lane & 7) == 0 && r < nrow && (on || pad)) ep.texp[gemm_exp_at(nc, p.mt, lr, (p.n0 + j) / kGemmK)] = (int8_t)k;
      }
      if (MODE != EPI_STORE && ep.tile && r < nrow && (on || pad))
        gemm_tile_store4(ep, p.mt, lr, p.n0 + j, GRAD ? o1 : o2, sc);
    }
  }
}

template <int NW, bool TILED, bool GATES>
__global__ void __launch_bounds__(kGemmThreads, 1) k_gemm_split(const __grid_constant__ GemmArgs g) {
  using C = GemmCfg<NW, TILED>;
  constexpr int ST = kGemmStages;
  extern __shared__ __align__(1024) char smem[];
  __shared__ __align__(8) uint64_t fulla[ST], fullb[ST], done[ST], accfree[ST], drained, zfree;
  __shared__ uint32_t tbase_s;
  __shared__ int abort_s;
  volatile int *abort = &abort_s;
  const int tid = threadIdx.x, warp = tc::warp_index(), lane = tid & 31;
  const int nc = (g.K + kGemmK - 1) / kGemmK;
  const int ntile = (g.N + NW - 1) / NW * g.mt0[g.ntypes];
  if (tid == 0) {
    for (int s = 0; s < ST; ++s) {
      tc::mbar_init(&fulla[s], 256);
      tc::mbar_init(&fullb[s], 1);
      tc::mbar_init(&done[s], 1);
      tc::mbar_init(&accfree[s], 256);
    }
    tc::mbar_init(&drained, 256);
    tc::mbar_init(&zfree, 256);
    abort_s = 0;
    tc::fence_mbar_init();
  }
  if (warp == 0) tc::tmem_alloc(&tbase_s, C::TM);
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tbase = tbase_s, smem_u = tc::smem_u32(smem);
  int s = 0;            // stage of the running chunk
  uint32_t ph = 0;      // parity of its use of the stage
  bool first = true;    // the stage has not been used before
  bool ok = true;
  auto next = [&]() {
    if (++s == ST) {
      s = 0;
      ph ^= 1;
      first = false;
    }
  };

  if (warp == 17) {
    // ================= weights: NW of the 128 rows of a stored tile per chunk
    if (tc::elect_one()) {
      int issued = 0;
      for (int tile = blockIdx.x; tile < ntile && ok; tile += gridDim.x) {
        const GemmTilePos p = gemm_tile<NW>(g, tile);
        const char *src = reinterpret_cast<const char *>(g.t[p.ti].B) + (size_t)(p.n0 / kGemmTile) * nc * kGemmChunk +
                          (p.n0 % kGemmTile) * 16;
        for (int c = 0; c < nc; ++c, src += kGemmChunk, next(), ++issued) {
          if (!first && !(ok = gemm_wait(&done[s], ph ^ 1, abort))) break;
          const uint32_t dst = smem_u + s * C::STAGE + C::AB;
          tc::mbar_arrive_expect_tx(&fullb[s], C::BB + (TILED ? C::AB : 0));
          if (TILED)
            tc::bulk_load(dst - C::AB, g.At + ((size_t)p.mt * nc + c) * (2 * kGemmPart), C::AB, &fullb[s]);
          if (NW == kGemmTile) {
            tc::bulk_load(dst, src, C::BB, &fullb[s]);
          } else {
#pragma unroll
            for (int q = 0; q < 12; ++q)
              tc::bulk_load(dst + q * NW * 16, src + q * kGemmTile * 16, NW * 16, &fullb[s]);
          }
        }
      }
      // copies still in flight (only after a give-up): the last ST issued chunks
      for (int c = issued > ST ? issued - ST : 0; c < issued; ++c) tc::mbar_wait(&fullb[c % ST], (c / ST) & 1);
    }
  } else if (warp == 16) {
    // ================= MMA issuer
    if (tc::elect_one()) {
      int last = -1;
      uint32_t last_ph = 0;
      for (int tile = blockIdx.x; tile < ntile && ok; tile += gridDim.x) {
        const GemmTilePos p = gemm_tile<NW>(g, tile);
        const uint32_t idesc = tc::idesc_f16(128, (p.nv + 15) / 16 * 16, 0, 0);
        for (int c = 0; c < nc; ++c, next()) {
          {  // the polls overlap (250 clocks each, one after the other)
            const bool r0 = first || tc::mbar_test(tc::smem_u32(&accfree[s]), ph ^ 1);
            const bool r1 = TILED || tc::mbar_test(tc::smem_u32(&fulla[s]), ph), r2 = tc::mbar_test(tc::smem_u32(&fullb[s]), ph);
            ok = (r0 || gemm_wait(&accfree[s], ph ^ 1, abort)) && (r1 || gemm_wait(&fulla[s], ph, abort)) &&
                 (r2 || gemm_wait(&fullb[s], ph, abort));
          }
          if (!ok) break;
          tc::fence_after_sync();
          const uint32_t a_u = smem_u + s * C::STAGE, b_u = a_u + C::AB, d = tbase + s * NW;
          const int nks = min(2, (g.K - c * kGemmK + 15) / 16);
#pragma unroll
          for (int q = 0; q < 4; ++q) {  // lo.hi, hi.lo2, hi.lo, hi.hi
            const uint32_t ap = a_u + (q == 0 ? 4 * C::ALBO : 0),
                           bp = b_u + (q == 1 ? 2 : q == 2 ? 1 : 0) * (4 * NW * 16);
#pragma unroll
            for (int ks = 0; ks < 2; ++ks)
              if (ks < nks)
                tc::mma_f16kind(d, tc::make_desc(ap + 2 * ks * C::ALBO, C::ALBO, 128),
                                tc::make_desc(bp + 2 * ks * NW * 16, NW * 16, 128), idesc,
                                (q > 0 || ks > 0) ? 1u : 0u);
          }
          tc::commit(&done[s]);
          last = s;
          last_ph = ph;
        }
      }
      if (last >= 0) tc::mbar_wait(&done[last], last_ph);  // the last MMAs complete before the CTA exits
    }
  } else if (!TILED && warp >= 8) {
    // ================= A: rows 16 w + 4 i + lane / 8, columns 4 (lane % 8) .. + 4: an
    // instruction loads four rows' whole lines.  (With 8 lanes on 8 rows' same
    // columns the line reads conflicted 8-way: 1,000 of a chunk's 2,000 clocks.)
    const int w = warp - 8, r4 = lane >> 3, k4 = 4 * (lane & 7);
    auto run = [&](auto vec) {  // vec: K, so every row's start, a multiple of 4
      // the chunk being loaded, PF ahead of the one being stored (in the next
      // tile where a tile has no more); loads are unconditional, from clamped
      // addresses (rows past the end are never stored; K past the end is zeroed
      // when it is split)
      constexpr int PF = 3;
      int lt = blockIdx.x, lc = 0;
      const float *arow[4] = {g.A, g.A, g.A, g.A};
      auto load = [&](float4 (&v)[4], float (&am)[4]) {
        if (lc == 0) {
          const GemmTilePos p = gemm_tile<NW>(g, lt);
          const GemmType &gt = g.t[p.ti];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int r = p.m0 + 16 * w + 4 * i + r4;
            const size_t at = r < gt.Mrows ? gt.rm.atom(r) : 0;
            arow[i] = g.A + at * (size_t)g.lda;
            am[i] = gt.gmax ? gt.gmax[at] : -gt.ascale;
          }
        }
        const int k = lc * kGemmK + k4;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float *a = arow[i];
          if constexpr (decltype(vec)::value)
            v[i] = *reinterpret_cast<const float4 *>(a + min(k, g.K - 4));
          else
            v[i] = make_float4(a[min(k, g.K - 1)], a[min(k + 1, g.K - 1)], a[min(k + 2, g.K - 1)],
                               a[min(k + 3, g.K - 1)]);
        }
        if (++lc == nc) {
          lc = 0;
          if (lt + (int)gridDim.x < ntile) lt += gridDim.x;
        }
      };
      float4 v[PF][4];
      float am[PF][4], asc[4] = {1.f, 1.f, 1.f, 1.f};
#pragma unroll
      for (int q = 0; q < PF; ++q) load(v[q], am[q]);
      int c = 0;
      auto chunk = [&](float4 (&v)[4], float (&am)[4]) {
        if (c == 0) {
#pragma unroll
          for (int i = 0; i < 4; ++i) asc[i] = am[i] < 0.f ? -am[i] : row_scale(am[i]);
        }
        if (++c == nc) {
          c = 0;
          const int k = (nc - 1) * kGemmK + k4;
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            if (k >= g.K) v[i].x = 0.f;
            if (k + 1 >= g.K) v[i].y = 0.f;
            if (k + 2 >= g.K) v[i].z = 0.f;
            if (k + 3 >= g.K) v[i].w = 0.f;
          }
        }
        if (!first && !gemm_wait(&done[s], ph ^ 1, abort)) ok = false;
        ok = __all_sync(0xffffffffu, ok);
        char *as = smem + s * C::STAGE + (lane >> 1 & 3) * C::ALBO + (16 * w + r4) * 16 + (lane & 1) * 8;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const tc::f2 sc = tc::pk1(asc[i]);
          uint2 h, l;
          tc::split_pair(tc::mul2(tc::pk(v[i].x, v[i].y), sc), h.x, l.x);
          tc::split_pair(tc::mul2(tc::pk(v[i].z, v[i].w), sc), h.y, l.y);
          *reinterpret_cast<uint2 *>(as + i * 64) = h;
          *reinterpret_cast<uint2 *>(as + 4 * C::ALBO + i * 64) = l;
        }
        tc::fence_proxy_async();
        tc::mbar_arrive(&fulla[s]);
        load(v, am);
        next();
      };
      const int total = (int)blockIdx.x < ntile ? (ntile - 1 - (int)blockIdx.x) / (int)gridDim.x * nc + nc : 0;
      for (int i = 0; i < total && ok; i += PF)
#pragma unroll
        for (int q = 0; q < PF; ++q)
          if (i + q < total && ok) chunk(v[q], am[q]);
    };
    if ((g.K & 3) == 0) run(std::true_type{});
    else run(std::false_type{});
  } else {
    // ================= sums and epilogue, of every tile or (TILED) of every
    // second one per group of 8 warps
    constexpr int EG = TILED ? 2 : 1;
    const int row = tid & 127, half = (tid >> 7) & 1, grp = warp >> 3;
    const uint32_t tl = tbase + ((uint32_t)((warp & 3) * 32) << 16) + half * (NW / 2);
    float *zs = reinterpret_cast<float *>(smem + ST * C::STAGE);
    int i = 0;
    for (int tile = blockIdx.x; tile < ntile && ok; tile += gridDim.x, ++i) {
      if (EG == 2 && (i & 1) != grp) {  // the other group's tile
        const int t = s + nc;
        ph ^= (uint32_t)(t / ST) & 1;
        s = t % ST;
        continue;
      }
      const GemmTilePos p = gemm_tile<NW>(g, tile);
      const GemmType &gt = g.t[p.ti];
      tc::f2 acc[NW / 4];
#pragma unroll
      for (int k = 0; k < NW / 4; ++k) acc[k] = tc::pk1(0.f);
      // scale exponents of eight chunks (a load per chunk, which the arrivals on accfree
      // wait for, made the six GEMMs of 98,304 atoms 10 % slower)
      const int2 *aexp = GATES ? reinterpret_cast<const int2 *>(g.Aexp + gemm_exp_at(nc, p.mt, row, 0)) : nullptr;
      int2 ew = GATES ? *aexp : make_int2(0, 0);
      // the other group has added all of the previous tile's sums: no stage's
      // barrier is more than one phase ahead of this group's wait
      if (EG == 2 && i > 0) ok = __all_sync(0xffffffffu, gemm_wait(&drained, (i - 1) & 1, abort));
      for (int c = 0; c < nc && ok; ++c, next()) {
        if (GATES && c > 0) {
          if ((c & 7) == 0) ew = aexp[c >> 3];
          else if ((c & 3) == 0) ew.x = ew.y;
          else ew.x >>= 8;
        }
        const float u = GATES ? pow2i(-(int)(int8_t)ew.x) : 1.f;
        ok = __all_sync(0xffffffffu, gemm_wait(&done[s], ph, abort));
        if (!ok) break;
        tc::fence_after_sync();
#pragma unroll
        for (int q = 0; q < NW / 2; q += 16) {
          uint32_t r[16];
          tc::tmem_ld16_issue(tl + s * NW + q, r);
          tc::tmem_wait();
#pragma unroll
          for (int k = 0; k < 8; ++k) {
            const tc::f2 x = tc::pk(__uint_as_float(r[2 * k]), __uint_as_float(r[2 * k + 1]));
            acc[q / 2 + k] = GATES ? tc::fma2(x, tc::pk1(u), acc[q / 2 + k]) : tc::add2(acc[q / 2 + k], x);
          }
        }
        tc::fence_before_sync();
        tc::mbar_arrive(&accfree[s]);
      }
      if (EG == 2) tc::mbar_arrive(&drained);
      // the previous tile's epilogue (the other group's) has read zs
      if (EG == 2 && i > 0 && ok) ok = __all_sync(0xffffffffu, gemm_wait(&zfree, (i - 1) & 1, abort));
      // through shared memory: rows by warps, columns by lanes
      {
        const int r = p.m0 + row;
        const float rs = (gt.gmax && r < gt.Mrows) ? row_scale(gt.gmax[gt.rm.atom(r)]) : gt.ascale;
        const float us = 1.f / (rs * gt.wscale);
        float *z = zs + row * C::ZS + half * (NW / 2);
#pragma unroll
        for (int i = 0; i < NW / 4; i += 2) {
          float4 v;
          tc::upk(acc[i], v.x, v.y);
          tc::upk(acc[i + 1], v.z, v.w);
          *reinterpret_cast<float4 *>(z + 2 * i) = make_float4(v.x * us, v.y * us, v.z * us, v.w * us);
        }
      }
      {  // zs written; every warp agrees on ok, so that they leave the tile loop together
        int all;
        asm volatile(
            "{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\tbar.red.and.pred q, %2, 256, p;\n\t"
            "selp.u32 %0, 1, 0, q;\n\t}"
            : "=r"(all)
            : "r"((uint32_t)ok), "r"(1 + grp)
            : "memory");
        ok = all != 0;
      }
      const float bad = ok ? 0.f : __int_as_float(0x7fffffff);  // a wait gave up: NaN results
      if constexpr (GATES) {
        if (gt.ep.mode == EPI_STORE) gemm_epilogue<NW, EPI_STORE>(gt, p, zs, bad);
        else if (gt.ep.mode == EPI_GRAD_RES) gemm_epilogue<NW, EPI_GRAD_RES>(gt, p, zs, bad);
        else gemm_epilogue<NW, EPI_GRAD>(gt, p, zs, bad);
      } else {
        if (gt.ep.mode == EPI_TANH) gemm_epilogue<NW, EPI_TANH>(gt, p, zs, bad);
        else gemm_epilogue<NW, EPI_TANH_RES>(gt, p, zs, bad);
      }
      // zs is free again; and every thread of the group has arrived on drained and
      // zfree before one of them waits there for a later phase
      if (EG == 2) tc::mbar_arrive(&zfree);
      asm volatile("bar.sync %0, 256;" ::"r"(1 + grp) : "memory");
    }
  }
  tc::fence_before_sync();
  __syncthreads();
  if (tid == 0 && abort_s) atomicOr(g.err, 1);  // a wait gave up (k_finalize)
  if (warp == 0) tc::tmem_dealloc(tbase, C::TM);
}

template <int NW, bool TILED, bool GATES>
static int launch_gemm_m(const GemmArgs &g, int nsm, cudaStream_t st) {
  const int smem = GemmCfg<NW, TILED>::SMEM;
  DPB_CUDA_TRY(cudaFuncSetAttribute(k_gemm_split<NW, TILED, GATES>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  const int ntile = (g.N + NW - 1) / NW * g.mt0[g.ntypes];
  k_gemm_split<NW, TILED, GATES><<<ntile < nsm ? ntile : nsm, kGemmThreads, smem, st>>>(g);
  count_launch();
  DPB_LAUNCH_CHECK();
  return DPB_OK;
}

template <int NW>
static int launch_gemm_w(const GemmArgs &g, int nsm, cudaStream_t st) {
  if (!g.At) return launch_gemm_m<NW, false, false>(g, nsm, st);
  return g.Aexp ? launch_gemm_m<NW, true, true>(g, nsm, st) : launch_gemm_m<NW, true, false>(g, nsm, st);
}

size_t gemm_exp_bytes(size_t rows, int K) { return rows * (((K + kGemmK - 1) / kGemmK + 7) & ~7); }
size_t gemm_operand_halves(int mt, int K) { return (size_t)mt * ((K + kGemmK - 1) / kGemmK) * (2 * kGemmPart); }

// Every centre type in one launch (g.t, g.mt0 filled).  128 columns per CTA keep
// the tensor core busiest; 64 and 32 where that leaves SMs without a CTA.
int launch_gemm_split(const GemmArgs &g, cudaStream_t st) {
  const int mt = g.mt0[g.ntypes];
  if (mt == 0) return DPB_OK;
  int dev = 0, nsm = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  const auto ctas = [&](int nw) { return (long long)((g.N + nw - 1) / nw) * mt; };
  if (ctas(128) >= nsm) return launch_gemm_w<128>(g, nsm, st);
  if (ctas(64) >= nsm) return launch_gemm_w<64>(g, nsm, st);
  return launch_gemm_w<32>(g, nsm, st);
}

}  // namespace dpb

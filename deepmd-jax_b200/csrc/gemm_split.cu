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
// and gates' from bounds known at model creation, the descriptor's per atom from
// its largest entry (gmax, written with G), all divided out of the sum exactly.
#include "internal.cuh"
#include "tc.cuh"

namespace dpb {

constexpr int kGemmK = 32;                            // K of one pipeline stage
constexpr int kGemmALbo = 128 * 16;                   // A: bytes between 8-wide K groups
constexpr int kGemmAB = 2 * 4 * kGemmALbo;            // A stage: hi, lo
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
// three stages (A, weights and a TMEM accumulator each):
//   warps 0-7   add each chunk's sum from TMEM to their registers (two threads
//               per row, half the columns each) and run the epilogue, while
//   warps 8-15  load A in FP32 four chunks ahead, split it and store the operand
//               (16-byte stores of 8 rows, no bank conflicts),
//   warp 16     issues the MMAs, and
//   warp 17     the bulk copies of the weights
// already work on the next tile.  (With every thread loading, adding and
// waiting in step, two CTAs per SM, a chunk took 2,200 clocks per SM against the
// 530 of its MMAs: 411 instructions per warp and chunk and three dependent waits.)
constexpr int kGemmStages = 3;
constexpr int kGemmThreads = 18 * 32;

template <int NW>
struct GemmCfg {
  static constexpr int BB = 3 * 4 * NW * 16, STAGE = kGemmAB + BB;
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
  int ti, m0, n0, nv;
};
template <int NW>
__device__ __forceinline__ GemmTilePos gemm_tile(const GemmArgs &g, int tile) {
  const int ntn = (g.N + NW - 1) / NW, mt = tile / ntn;
  GemmTilePos p;
  p.n0 = (tile - mt * ntn) * NW;
  p.nv = min(NW, g.N - p.n0);
  p.ti = 0;
#pragma unroll
  for (int t = 1; t < kMaxTypes; ++t)
    if (t < g.ntypes && mt >= g.mt0[t]) p.ti = t;
  p.m0 = (mt - g.mt0[p.ti]) * 128;
  return p;
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
  constexpr int ZS = GemmCfg<NW>::ZS, LQ = NW / 4, RPW = 32 / LQ;  // lanes per row, rows per warp pass
  constexpr int RB = MODE == EPI_STORE ? 4 : 2;
  constexpr bool TANH = MODE == EPI_TANH || MODE == EPI_TANH_RES, GRAD = MODE == EPI_GRAD || MODE == EPI_GRAD_RES;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const Epi &ep = gt.ep;
  if ((ep.ld & 3) != 0) {
    for (int lr = warp; lr < 128 && p.m0 + lr < gt.Mrows; lr += 8) {
      const size_t at = gt.rm.atom(p.m0 + lr) * (size_t)ep.ld + p.n0;
      for (int j = lane; j < p.nv; j += 32) {
        const int n = p.n0 + j;
        const float *am = MODE == EPI_TANH_RES ? ep.hprev : ep.gmat;
        const float a = GRAD && ep.gvec ? ep.gvec[n] : (MODE == EPI_TANH_RES || GRAD) && am ? am[at + j] : 0.f;
        float o1 = 0.f, o2 = 0.f;
        gemm_epi1<MODE>(zs[lr * ZS + j] + bad, TANH ? ep.bias[n] : 0.f,
                        MODE == EPI_TANH_RES || MODE == EPI_GRAD_RES ? ep.dt[n] : 1.f, a, GRAD ? ep.tin[at + j] : 0.f,
                        o1, o2);
        ep.out1[at + j] = o1;
        if (MODE == EPI_TANH_RES || MODE == EPI_GRAD_RES || (MODE == EPI_TANH && ep.out2)) ep.out2[at + j] = o2;
      }
    }
    return;
  }
  const int j = 4 * (lane % LQ), rl = lane / LQ;
  const bool on = j < p.nv;
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
  auto ld4 = [&](const float *q) { return on ? *reinterpret_cast<const float4 *>(q) : zero; };
  const float4 bias = TANH ? ld4(ep.bias + p.n0 + j) : zero;
  const float4 dt = MODE == EPI_TANH_RES || MODE == EPI_GRAD_RES ? ld4(ep.dt + p.n0 + j) : zero;
  const float4 gv = GRAD && ep.gvec ? ld4(ep.gvec + p.n0 + j) : zero;
  const float *am = MODE == EPI_TANH_RES ? ep.hprev : GRAD && !ep.gvec ? ep.gmat : nullptr;
#pragma unroll 1
  for (int q = 0; q < 16; q += RB * RPW) {
    float4 x[RB], a[RB], t[RB];
    size_t at[RB];
    bool act[RB];
#pragma unroll
    for (int b = 0; b < RB; ++b) {
      const int lr = 16 * warp + q + b * RPW + rl;
      act[b] = on && p.m0 + lr < gt.Mrows;
      at[b] = act[b] ? gt.rm.atom(p.m0 + lr) * (size_t)ep.ld + p.n0 + j : 0;
      a[b] = gv;
      t[b] = zero;
      if (act[b]) {
        if ((MODE == EPI_TANH_RES || GRAD) && am) a[b] = *reinterpret_cast<const float4 *>(am + at[b]);
        if (GRAD) t[b] = *reinterpret_cast<const float4 *>(ep.tin + at[b]);
      }
      x[b] = *reinterpret_cast<const float4 *>(zs + lr * ZS + j);
    }
#pragma unroll
    for (int b = 0; b < RB; ++b) {
      if (!act[b]) continue;
      float4 o1 = zero, o2 = zero;
      gemm_epi1<MODE>(x[b].x + bad, bias.x, dt.x, a[b].x, t[b].x, o1.x, o2.x);
      gemm_epi1<MODE>(x[b].y + bad, bias.y, dt.y, a[b].y, t[b].y, o1.y, o2.y);
      gemm_epi1<MODE>(x[b].z + bad, bias.z, dt.z, a[b].z, t[b].z, o1.z, o2.z);
      gemm_epi1<MODE>(x[b].w + bad, bias.w, dt.w, a[b].w, t[b].w, o1.w, o2.w);
      *reinterpret_cast<float4 *>(ep.out1 + at[b]) = o1;
      if (MODE == EPI_TANH_RES || MODE == EPI_GRAD_RES || (MODE == EPI_TANH && ep.out2))
        *reinterpret_cast<float4 *>(ep.out2 + at[b]) = o2;
    }
  }
}

template <int NW>
__global__ void __launch_bounds__(kGemmThreads, 1) k_gemm_split(const __grid_constant__ GemmArgs g) {
  using C = GemmCfg<NW>;
  constexpr int ST = kGemmStages;
  extern __shared__ __align__(1024) char smem[];
  __shared__ __align__(8) uint64_t fulla[ST], fullb[ST], done[ST], accfree[ST];
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
          const uint32_t dst = smem_u + s * C::STAGE + kGemmAB;
          tc::mbar_arrive_expect_tx(&fullb[s], C::BB);
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
          ok = (first || gemm_wait(&accfree[s], ph ^ 1, abort)) && gemm_wait(&fulla[s], ph, abort) &&
               gemm_wait(&fullb[s], ph, abort);
          if (!ok) break;
          tc::fence_after_sync();
          const uint32_t a_u = smem_u + s * C::STAGE, b_u = a_u + kGemmAB, d = tbase + s * NW;
          const int nks = min(2, (g.K - c * kGemmK + 15) / 16);
#pragma unroll
          for (int q = 0; q < 4; ++q) {  // lo.hi, hi.lo2, hi.lo, hi.hi
            const uint32_t ap = a_u + (q == 0 ? 4 * kGemmALbo : 0),
                           bp = b_u + (q == 1 ? 2 : q == 2 ? 1 : 0) * (4 * NW * 16);
#pragma unroll
            for (int ks = 0; ks < 2; ++ks)
              if (ks < nks)
                tc::mma_f16kind(d, tc::make_desc(ap + 2 * ks * kGemmALbo, kGemmALbo, 128),
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
  } else if (warp >= 8) {
    // ================= A: rows 16 w + 8 i + lane % 8, K group lane / 8 of 8 values
    const int w = warp - 8, r8 = lane & 7, k8 = lane >> 3;
    const bool vec = (g.lda & 3) == 0;
    for (int tile = blockIdx.x; tile < ntile && ok; tile += gridDim.x) {
      const GemmTilePos p = gemm_tile<NW>(g, tile);
      const GemmType &gt = g.t[p.ti];
      const float *arow[2];
      float asc[2];
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int r = p.m0 + 16 * w + 8 * i + r8;
        const size_t at = r < gt.Mrows ? gt.rm.atom(r) : 0;
        arow[i] = r < gt.Mrows ? g.A + at * (size_t)g.lda : nullptr;
        asc[i] = gt.gmax ? row_scale(gt.gmax[at]) : gt.ascale;
      }
      auto load = [&](int c, float4 (&v)[4]) {
        const int k = c * kGemmK + 8 * k8;
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          v[2 * i] = v[2 * i + 1] = make_float4(0.f, 0.f, 0.f, 0.f);
          if (arow[i] == nullptr || c >= nc) continue;
          const float *a = arow[i] + k;
          if (vec && k + 7 < g.K) {
            v[2 * i] = *reinterpret_cast<const float4 *>(a);
            v[2 * i + 1] = *reinterpret_cast<const float4 *>(a + 4);
          } else {
            float t[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) t[e] = k + e < g.K ? a[e] : 0.f;
            v[2 * i] = make_float4(t[0], t[1], t[2], t[3]);
            v[2 * i + 1] = make_float4(t[4], t[5], t[6], t[7]);
          }
        }
      };
      float4 v[4][4];  // four chunks in flight: the loads' latency is about two chunks' MMAs
#pragma unroll
      for (int q = 0; q < 4; ++q) load(q, v[q]);
      auto chunk = [&](int c, float4 (&v)[4]) {
        if (!first && !gemm_wait(&done[s], ph ^ 1, abort)) ok = false;
        ok = __all_sync(0xffffffffu, ok);
        char *as = smem + s * C::STAGE + k8 * kGemmALbo + (16 * w + r8) * 16;
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const tc::f2 sc = tc::pk1(asc[i]);
          uint32_t h[4], l[4];
          tc::split_pair(tc::mul2(tc::pk(v[2 * i].x, v[2 * i].y), sc), h[0], l[0]);
          tc::split_pair(tc::mul2(tc::pk(v[2 * i].z, v[2 * i].w), sc), h[1], l[1]);
          tc::split_pair(tc::mul2(tc::pk(v[2 * i + 1].x, v[2 * i + 1].y), sc), h[2], l[2]);
          tc::split_pair(tc::mul2(tc::pk(v[2 * i + 1].z, v[2 * i + 1].w), sc), h[3], l[3]);
          *reinterpret_cast<uint4 *>(as + i * 128) = make_uint4(h[0], h[1], h[2], h[3]);
          *reinterpret_cast<uint4 *>(as + 4 * kGemmALbo + i * 128) = make_uint4(l[0], l[1], l[2], l[3]);
        }
        load(c + 4, v);
        tc::fence_proxy_async();
        tc::mbar_arrive(&fulla[s]);
        next();
      };
      for (int c = 0; c < nc && ok; c += 4)
#pragma unroll
        for (int q = 0; q < 4; ++q)
          if (c + q < nc && ok) chunk(c + q, v[q]);
    }
  } else {
    // ================= sums and epilogue
    const int row = tid & 127, half = tid >> 7;
    const uint32_t tl = tbase + ((uint32_t)((warp & 3) * 32) << 16) + half * (NW / 2);
    float *zs = reinterpret_cast<float *>(smem + ST * C::STAGE);
    for (int tile = blockIdx.x; tile < ntile && ok; tile += gridDim.x) {
      const GemmTilePos p = gemm_tile<NW>(g, tile);
      const GemmType &gt = g.t[p.ti];
      tc::f2 acc[NW / 4];
#pragma unroll
      for (int i = 0; i < NW / 4; ++i) acc[i] = tc::pk1(0.f);
      for (int c = 0; c < nc; ++c, next()) {
        ok = __all_sync(0xffffffffu, gemm_wait(&done[s], ph, abort));
        if (!ok) break;
        tc::fence_after_sync();
#pragma unroll
        for (int q = 0; q < NW / 2; q += 16) {
          uint32_t r[16];
          tc::tmem_ld16_issue(tl + s * NW + q, r);
          tc::tmem_wait();
#pragma unroll
          for (int i = 0; i < 8; ++i)
            acc[q / 2 + i] =
                tc::add2(acc[q / 2 + i], tc::pk(__uint_as_float(r[2 * i]), __uint_as_float(r[2 * i + 1])));
        }
        tc::fence_before_sync();
        tc::mbar_arrive(&accfree[s]);
      }
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
            "{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\tbar.red.and.pred q, 1, 256, p;\n\t"
            "selp.u32 %0, 1, 0, q;\n\t}"
            : "=r"(all)
            : "r"((uint32_t)ok)
            : "memory");
        ok = all != 0;
      }
      const float bad = ok ? 0.f : __int_as_float(0x7fffffff);  // a wait gave up: NaN results
      switch (gt.ep.mode) {
        case EPI_STORE: gemm_epilogue<NW, EPI_STORE>(gt, p, zs, bad); break;
        case EPI_TANH: gemm_epilogue<NW, EPI_TANH>(gt, p, zs, bad); break;
        case EPI_TANH_RES: gemm_epilogue<NW, EPI_TANH_RES>(gt, p, zs, bad); break;
        case EPI_GRAD_RES: gemm_epilogue<NW, EPI_GRAD_RES>(gt, p, zs, bad); break;
        case EPI_GRAD: gemm_epilogue<NW, EPI_GRAD>(gt, p, zs, bad); break;
      }
      asm volatile("bar.sync 1, 256;" ::: "memory");  // zs is free again
    }
  }
  tc::fence_before_sync();
  __syncthreads();
  if (warp == 0) tc::tmem_dealloc(tbase, C::TM);
}

template <int NW>
static int launch_gemm_w(const GemmArgs &g, int nsm, cudaStream_t st) {
  const int smem = GemmCfg<NW>::SMEM;
  DPB_CUDA_TRY(cudaFuncSetAttribute(k_gemm_split<NW>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  const int ntile = (g.N + NW - 1) / NW * g.mt0[g.ntypes];
  k_gemm_split<NW><<<ntile < nsm ? ntile : nsm, kGemmThreads, smem, st>>>(g);
  count_launch();
  DPB_LAUNCH_CHECK();
  return DPB_OK;
}

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

// Mixed-precision (FP16 tensor-core) evaluation path.
#include "rows.cuh"

namespace dpb {

// ---------------------------------------------------------------- self-test
// Known-answer test of the tcgen05 path: D(128x64) = A(128x32) B(32x64) with
// A[m][k] = ((m*3 + k*5) % 17 - 8) / 8, B[k][n] = ((k*7 + n*11) % 13 - 6) / 4
// (all exact in bf16).  variant 0: A and B K-major; 1: A and B MN-major.
// Writes D row-major to out; err gets 1 on an mbarrier timeout.
__global__ void __launch_bounds__(128) k_selftest_umma(int variant, float *out, int *err) {
  constexpr int M = 128, N = 64, K = 32;
  __shared__ __align__(128) __nv_bfloat16 As[M * K];
  __shared__ __align__(128) __nv_bfloat16 Bs[N * K];
  __shared__ __align__(8) uint64_t mbar;
  __shared__ uint32_t tbase;
  const int tid = threadIdx.x;
  char *Ab = reinterpret_cast<char *>(As), *Bb = reinterpret_cast<char *>(Bs);
  for (int e = tid; e < M * K; e += 128) {
    const int m = e / K, k = e % K;
    const float v = (float)((m * 3 + k * 5) % 17 - 8) / 8.f;
    const uint32_t off = variant == 0 ? tc::kmajor_off(m, k, K) : tc::mnmajor_off(k, m, M);
    *reinterpret_cast<__nv_bfloat16 *>(Ab + off) = __float2bfloat16_rn(v);
  }
  for (int e = tid; e < N * K; e += 128) {
    const int k = e / N, n = e % N;
    const float v = (float)((k * 7 + n * 11) % 13 - 6) / 4.f;
    const uint32_t off = variant == 0 ? tc::kmajor_off(n, k, K) : tc::mnmajor_off(k, n, N);
    *reinterpret_cast<__nv_bfloat16 *>(Bb + off) = __float2bfloat16_rn(v);
  }
  if (tid == 0) tc::mbar_init(&mbar, 1);
  if (tid < 32) tc::tmem_alloc(&tbase, 64);
  tc::fence_proxy_async();
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t d = tbase;
  if (tid == 0) {
    const uint32_t idesc = tc::idesc_bf16(M, N, variant, variant);
    const uint32_t a0 = tc::smem_u32(As), b0 = tc::smem_u32(Bs);
    for (int ks = 0; ks < K / 16; ++ks) {
      uint64_t ad, bd;
      if (variant == 0) {
        ad = tc::make_desc(a0 + tc::kmajor_off(0, ks * 16, K), 128, (K / 8) * 128);
        bd = tc::make_desc(b0 + tc::kmajor_off(0, ks * 16, K), 128, (K / 8) * 128);
      } else {
        ad = tc::make_desc(a0 + tc::mnmajor_off(ks * 16, 0, M), (M / 8) * 128, 128);
        bd = tc::make_desc(b0 + tc::mnmajor_off(ks * 16, 0, N), (N / 8) * 128, 128);
      }
      tc::mma_f16kind(d, ad, bd, idesc, ks > 0);
    }
    tc::commit(&mbar);
  }
  if (!tc::mbar_wait(&mbar, 0)) atomicOr(err, 1);
  tc::fence_after_sync();
  const int warp = tid >> 5;
  for (int c = 0; c < N; c += 16) {
    float v[16];
    tc::tmem_ld16(d + ((uint32_t)(warp * 32) << 16) + c, v);
    for (int i = 0; i < 16; ++i) out[tid * N + c + i] = v[i];
  }
  tc::fence_before_sync();
  __syncthreads();
  if (tid < 32) tc::tmem_dealloc(d, 64);
}

// ---------------------------------------------------------------- shared pieces
// Tile geometry of one embedding net E0 -> E1 -> E2 on the tensor cores.  The
// operands are FP16 (10 mantissa bits, against BF16's 7; every embedding
// activation is a sum of at most three tanh values, far inside FP16's range).
// The A operands of layers 1 and 2 carry a ones column at K index E0 (E1) and
// the B tiles hold the layer's bias in that K row, so the MMA adds the bias.
__host__ __device__ constexpr int imax(int a, int b) { return a > b ? a : b; }
__host__ __device__ constexpr int imin(int a, int b) { return a < b ? a : b; }

template <int E0, int E1, int E2>
struct MixDims {
  static constexpr int K1 = (E0 + 1 + 15) / 16 * 16;  // layer-1 K: inputs and the ones column
  static constexpr int N1 = (E1 + 15) / 16 * 16;
  static constexpr int K2 = (E1 + 1 + 15) / 16 * 16;
  static constexpr int N2 = (E2 + 15) / 16 * 16;
  static constexpr int W1B = N1 * K1 * 2;  // bytes of the layer-1 B tile (K-major)
  static constexpr int W2B = N2 * K2 * 2;  // bytes of the layer-2 B tile (K-major)
  static constexpr int NETB = W1B + W2B;
  static constexpr int NSMALL = (2 * E0 + 3) / 4 * 4;  // w0, b0 (fp32)
  static constexpr int OPA_A0 = 128 * K1 * 2, OPA_A1 = 128 * K2 * 2, OPA_H2 = 128 * N2 * 2;
  static constexpr int OPA = imax(OPA_A0, imax(OPA_A1, OPA_H2));
  static constexpr int Z1 = E1 / E0, Z2 = E2 / E1;
  static_assert(Z1 * E0 == E1 && Z2 * E1 == E2 && Z1 >= 1 && Z1 <= 2 && Z2 >= 1 && Z2 <= 2,
                "residual ratios 1 or 2");
  static_assert(E1 % 2 == 0 && E2 % 2 == 0 && N1 <= 64 && N2 <= 128, "tile widths");
};

// Column split between the two threads of a row ("halves", tid / 128): half
// 0 owns h1 columns [0, S1) and h2 columns [0, S2), half 1 the rest, with
// S2 = S1 * Z2 so every residual source h1[c / Z2] of a half's h2 columns is
// one of its own h1 columns; the A0 operand is split at A0C, A1 at S1, H2 at
// S2.  Half 0 computes h0 on [0, H0HI0), half 1 on [H0LO1, E0): the operand
// columns it writes and the residual sources of its h1 columns.
template <int E0, int E1, int E2>
struct HalfSplit {
  using MD = MixDims<E0, E1, E2>;
  static constexpr int S1 = (E1 / 2) / 8 * 8;
  static constexpr int S2 = S1 * MD::Z2;
  static constexpr int A0C = MD::K1 / 2;
  static constexpr int H0HI0 = imax(imin(A0C, E0), S1 / MD::Z1);
  static constexpr int H0LO1 = imin(A0C, S1 / MD::Z1);
  static constexpr int NP0 = imax((H0HI0 + 1) / 2, (E0 - H0LO1 + 1) / 2);  // h0 pairs per half
  static constexpr int NP1 = imax(S1 / 2, (E1 - S1 + 1) / 2);              // h1 pairs per half
  static_assert(S1 % 8 == 0 && S2 % 8 == 0 && H0LO1 % 2 == 0 && A0C % 8 == 0, "pair-aligned split");
};

// Asynchronous copy of one net's shared-memory image (FP16 B tiles and the
// FP32 first layer / biases); completes at the caller's cp_async_wait.
template <int E0, int E1, int E2>
__device__ __forceinline__ void mix_load_net(const DevModel &M, int k, char *netb, float *small) {
  using D = MixDims<E0, E1, E2>;
  const char *img = M.net_img[k];
  for (int e = threadIdx.x; e < D::NETB / 16; e += blockDim.x) tc::cp_async16(netb + 16 * e, img + 16 * e);
  const float *sm = M.net_small[k];
  for (int e = threadIdx.x; e < D::NSMALL / 4; e += blockDim.x) tc::cp_async16(small + 4 * e, sm + 4 * e);
  tc::cp_async_commit();
}

// Row geometry of the mixed form: the guarded norm, s(r) of utils.py:29-32
// and ds/dr as in row_geom, with fast reciprocals (a few ulp; the FP16 GEMMs
// downstream round far more).
__device__ __forceinline__ void row_geom_mixed(float3 x, float rcut, RowGeom &g) {
  g.x[0] = x.x; g.x[1] = x.y; g.x[2] = x.z;
  const float gx = fabsf(x.x) > 1e-15f ? x.x : 1e-15f;
  const float gy = fabsf(x.y) > 1e-15f ? x.y : 1e-15f;
  const float gz = fabsf(x.z) > 1e-15f ? x.z : 1e-15f;
  const float r = sqrtf(gx * gx + gy * gy + gz * gz);
  g.r = r;
  const float t = __fdividef(r, rcut);
  const float poly = 1.f - 3.f * t * t + 2.f * t * t * t;
  const float den = r + 1e-15f, inv_den = __fdividef(1.f, den);
  const bool in = (r > 1e-14f) && (t < 1.f);
  g.s = in ? poly * inv_den : 0.f;
  const float dpoly = __fdividef(-6.f * t + 6.f * t * t, rcut);
  g.dsdr = in ? (dpoly * den - poly) * inv_den * inv_den : 0.f;
}

// Adjoint of the row (row_adjoint) with fast reciprocals, for the mixed form.
__device__ __forceinline__ void row_adjoint_mixed(const RowGeom &g, float inv_std, const float gR[10], float gst,
                                                  float gx[3]) {
  const float inv_rp = __fdividef(1.f, g.r + 1e-16f);
  const float xh0 = g.x[0] * inv_rp, xh1 = g.x[1] * inv_rp, xh2 = g.x[2] * inv_rp;
  const float sn = g.s * inv_std;
  const float g_sn = gR[0] + kSqrt3 * (gR[1] * xh0 + gR[2] * xh1 + gR[3] * xh2) +
                     3.f * (gR[4] * (xh0 * xh0 - (1.f / 3.f)) + gR[5] * (xh1 * xh1 - (1.f / 3.f)) +
                            gR[6] * (xh2 * xh2 - (1.f / 3.f))) +
                     3.f * kSqrt2 * (gR[7] * xh0 * xh2 + gR[8] * xh1 * xh0 + gR[9] * xh2 * xh1);
  const float gh0 = sn * (kSqrt3 * gR[1] + 6.f * gR[4] * xh0 + 3.f * kSqrt2 * (gR[7] * xh2 + gR[8] * xh1));
  const float gh1 = sn * (kSqrt3 * gR[2] + 6.f * gR[5] * xh1 + 3.f * kSqrt2 * (gR[8] * xh0 + gR[9] * xh2));
  const float gh2 = sn * (kSqrt3 * gR[3] + 6.f * gR[6] * xh2 + 3.f * kSqrt2 * (gR[7] * xh0 + gR[9] * xh1));
  const float g_s = (g_sn + gst) * inv_std;
  const float g_r = g_s * g.dsdr - (gh0 * g.x[0] + gh1 * g.x[1] + gh2 * g.x[2]) * inv_rp * inv_rp;
  const float inv_r = __fdividef(1.f, g.r);
  const float d0 = fabsf(g.x[0]) > 1e-15f ? g.x[0] * inv_r : 0.f;
  const float d1 = fabsf(g.x[1]) > 1e-15f ? g.x[1] * inv_r : 0.f;
  const float d2 = fabsf(g.x[2]) > 1e-15f ? g.x[2] * inv_r : 0.f;
  gx[0] = gh0 * inv_rp + g_r * d0;
  gx[1] = gh1 * inv_rp + g_r * d1;
  gx[2] = gh2 * inv_rp + g_r * d2;
}

// Geometry of a compacted row (its relative coordinate) and the 10-channel
// env row (FP32).
__device__ __forceinline__ void mix_row_env(float4 rb, float rcut, float inv_std, float mean, RowGeom &gm, float &st,
                                            float R[10]) {
  row_geom_mixed(make_float3(rb.x, rb.y, rb.z), rcut, gm);
  const float sn = gm.s * inv_std;
  st = (gm.s - mean) * inv_std;
  const float inv_rp = __fdividef(1.f, gm.r + 1e-16f);
  const float xh[3] = {gm.x[0] * inv_rp, gm.x[1] * inv_rp, gm.x[2] * inv_rp};
  env_row(sn, xh, R);
}

// 8 floats times s as FP16, round to nearest, saturating at the largest
// finite FP16 value.
__device__ __forceinline__ uint4 pack8h(const float *v, float s) {
  return make_uint4(tc::as_u32(tc::f2_to_h2(v[0] * s, v[1] * s)), tc::as_u32(tc::f2_to_h2(v[2] * s, v[3] * s)),
                    tc::as_u32(tc::f2_to_h2(v[4] * s, v[5] * s)), tc::as_u32(tc::f2_to_h2(v[6] * s, v[7] * s)));
}

// ---------------------------------------------------------------- embedding rows in packed FP16
// The per-row epilogues of both embedding kernels work on pairs of adjacent
// columns packed in one register (__half2): tanh in FP32 (one MUFU operation
// per column) rounded to FP16, HADD2 for the residual, HFMA2 for the tangent
// (1 - t^2) dz + d_prev of the adjoint's forward-mode recompute, 1 - t^2 from the
// FP32 tanh.  A pair
// (c, c + 1) with c even; its residual source (utils.py:115-123, x_prev =
// repeat(x, Z)) is the pair (c, c + 1) of the layer below when Z = 1 and
// column c / 2, broadcast to both halves, when Z = 2.

// residual source pair of the even column c from the pairs `src` of the layer
// below, which start at column lo (compile-time indices after unrolling)
template <int Z>
__device__ __forceinline__ __half2 res_pair(const __half2 *src, int c, int lo) {
  if (Z == 1) return src[(c - lo) >> 1];
  const int k = (c >> 1) - lo;
  return (k & 1) ? __high2half2(src[k >> 1]) : __low2half2(src[k >> 1]);
}

// Operand pair of columns (c, c + 1) of a layer with E real columns whose
// pairs start at column lo: the values, the ones column at K index E (VALUE),
// zeros beyond.
template <int E, bool VALUE>
__device__ __forceinline__ __half2 operand_pair(const __half2 *p, int c, int lo) {
  const __half one = __float2half_rn(VALUE ? 1.f : 0.f), zero = __float2half_rn(0.f);
  if (c + 1 < E) return p[(c - lo) >> 1];
  if (c + 1 == E) return __halves2half2(__low2half(p[(c - lo) >> 1]), one);
  if (c == E) return __halves2half2(one, zero);
  return __halves2half2(zero, zero);
}

__device__ __forceinline__ void st_pairs(char *dst, __half2 a, __half2 b, __half2 c, __half2 d) {
  *reinterpret_cast<uint4 *>(dst) = make_uint4(tc::as_u32(a), tc::as_u32(b), tc::as_u32(c), tc::as_u32(d));
}

// Layer 0 (1 -> E0) of one half, FP32 pre-activation then FP16 pairs:
// h0 = tanh(s~ w0 + b0), with TANGENT also dh0/ds~ = (1 - h0^2) w0; writes
// the half's K-major A0 chunks (value operand a0, tangent operand a0t).
template <int E0, int E1, int E2, int HALF, bool TANGENT>
__device__ __forceinline__ void emb_layer0(float st, const float *sm, int row, char *a0, char *a0t,
                                           __half2 (&h0)[HalfSplit<E0, E1, E2>::NP0],
                                           __half2 (&d0)[HalfSplit<E0, E1, E2>::NP0]) {
  using MD = MixDims<E0, E1, E2>;
  using SP = HalfSplit<E0, E1, E2>;
  constexpr int lo = HALF ? SP::H0LO1 : 0, hi = HALF ? E0 : SP::H0HI0;
#pragma unroll
  for (int j = 0; j < (hi - lo + 1) / 2; ++j) {
    const int c = lo + 2 * j;
    const float za = fmaf(st, sm[c], sm[E0 + c]);
    const float zb = (c + 1 < E0) ? fmaf(st, sm[c + 1], sm[E0 + c + 1]) : 0.f;
    const float ta = tc::tanh_fast(za), tb = tc::tanh_fast(zb);
    const __half2 t = tc::f2_to_h2(ta, tb);
    h0[j] = t;
    if (TANGENT)
      d0[j] = tc::f2_to_h2(fmaf(-ta, ta, 1.f) * sm[c], (c + 1 < E0) ? fmaf(-tb, tb, 1.f) * sm[c + 1] : 0.f);
  }
  constexpr int c0 = HALF ? SP::A0C : 0, c1 = HALF ? MD::K1 : SP::A0C;
#pragma unroll
  for (int k8 = c0; k8 < c1; k8 += 8) {
    const uint32_t o = tc::kmajor_off(row, k8, MD::K1);
    st_pairs(a0 + o, operand_pair<E0, true>(h0, k8, lo), operand_pair<E0, true>(h0, k8 + 2, lo),
             operand_pair<E0, true>(h0, k8 + 4, lo), operand_pair<E0, true>(h0, k8 + 6, lo));
    if (TANGENT)
      st_pairs(a0t + o, operand_pair<E0, false>(d0, k8, lo), operand_pair<E0, false>(d0, k8 + 2, lo),
               operand_pair<E0, false>(d0, k8 + 4, lo), operand_pair<E0, false>(d0, k8 + 6, lo));
  }
}

// Layer 1 epilogue of one half: h1 = tanh(D1) + rep(h0) from the TMEM
// accumulator at tD (bias included), with TANGENT dh1 = (1 - t^2) D1t +
// rep(dh0) from tDt; 8 accumulator columns per TMEM load; writes the half's
// A1 chunks.
template <int E0, int E1, int E2, int HALF, bool TANGENT>
__device__ __forceinline__ void emb_epi1(uint32_t tD, uint32_t tDt, int row, char *a1, char *a1t,
                                         const __half2 (&h0)[HalfSplit<E0, E1, E2>::NP0],
                                         const __half2 (&d0)[HalfSplit<E0, E1, E2>::NP0],
                                         __half2 (&h1)[HalfSplit<E0, E1, E2>::NP1],
                                         __half2 (&d1)[HalfSplit<E0, E1, E2>::NP1]) {
  using MD = MixDims<E0, E1, E2>;
  using SP = HalfSplit<E0, E1, E2>;
  constexpr int c0 = HALF ? SP::S1 : 0, c1 = HALF ? E1 : SP::S1, h0lo = HALF ? SP::H0LO1 : 0;
#pragma unroll
  for (int g = c0 / 8 * 8; g < c1; g += 8) {
    uint32_t z[8], dz[8];
    tc::tmem_ld8_issue(tD + g, z);
    if (TANGENT) tc::tmem_ld8_issue(tDt + g, dz);
    tc::tmem_wait();
#pragma unroll
    for (int i = 0; i < 8; i += 2) {
      const int c = g + i;
      if (c < c0 || c >= c1) continue;
      const float ta = tc::tanh_fast(__uint_as_float(z[i])), tb = tc::tanh_fast(__uint_as_float(z[i + 1]));
      const __half2 t = tc::f2_to_h2(ta, tb);
      h1[(c - c0) >> 1] = __hadd2(t, res_pair<MD::Z1>(h0, c, h0lo));
      if (TANGENT) {
        const __half2 u = tc::f2_to_h2(fmaf(-ta, ta, 1.f), fmaf(-tb, tb, 1.f));
        d1[(c - c0) >> 1] = __hfma2(u, tc::f2_to_h2(__uint_as_float(dz[i]), __uint_as_float(dz[i + 1])),
                                    res_pair<MD::Z1>(d0, c, h0lo));
      }
    }
  }
  constexpr int k0 = HALF ? SP::S1 : 0, k1 = HALF ? MD::K2 : SP::S1;
#pragma unroll
  for (int k8 = k0; k8 < k1; k8 += 8) {
    const uint32_t o = tc::kmajor_off(row, k8, MD::K2);
    st_pairs(a1 + o, operand_pair<E1, true>(h1, k8, c0), operand_pair<E1, true>(h1, k8 + 2, c0),
             operand_pair<E1, true>(h1, k8 + 4, c0), operand_pair<E1, true>(h1, k8 + 6, c0));
    if (TANGENT)
      st_pairs(a1t + o, operand_pair<E1, false>(d1, k8, c0), operand_pair<E1, false>(d1, k8 + 2, c0),
               operand_pair<E1, false>(d1, k8 + 4, c0), operand_pair<E1, false>(d1, k8 + 6, c0));
  }
}

// Layer 2 epilogue of one half: h2 = tanh(D2) + rep(h1) (and with TANGENT
// dh2) for the half's columns (split at S2), zero past E2, stored per
// 8-column chunk at h2 + off(chunk) (and h2t + off(chunk)); OFF maps a column
// to the byte offset of the row's chunk in the operand layout the caller uses.
template <int E0, int E1, int E2, int HALF, bool TANGENT, typename OFF>
__device__ __forceinline__ void emb_epi2(uint32_t tD, uint32_t tDt, char *h2, char *h2t, OFF off,
                                         const __half2 (&h1)[HalfSplit<E0, E1, E2>::NP1],
                                         const __half2 (&d1)[HalfSplit<E0, E1, E2>::NP1]) {
  using MD = MixDims<E0, E1, E2>;
  using SP = HalfSplit<E0, E1, E2>;
  constexpr int c0 = HALF ? SP::S2 : 0, c1 = HALF ? MD::N2 : SP::S2, h1lo = HALF ? SP::S1 : 0;
  const __half2 zero2 = __float2half2_rn(0.f);
#pragma unroll
  for (int k8 = c0; k8 < c1; k8 += 8) {
    uint32_t z[8], dz[8];
    if (k8 < E2) {  // chunks past E2 are zero padding
      tc::tmem_ld8_issue(tD + k8, z);
      if (TANGENT) tc::tmem_ld8_issue(tDt + k8, dz);
      tc::tmem_wait();
    }
    __half2 hv[4], dv[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int c = k8 + 2 * u, i = 2 * u;
      hv[u] = dv[u] = zero2;
      if (c < E2) {
        const float ta = tc::tanh_fast(__uint_as_float(z[i])), tb = tc::tanh_fast(__uint_as_float(z[i + 1]));
        const __half2 t = tc::f2_to_h2(ta, tb);
        hv[u] = __hadd2(t, res_pair<MD::Z2>(h1, c, h1lo));
        if (TANGENT)
          dv[u] = __hfma2(tc::f2_to_h2(fmaf(-ta, ta, 1.f), fmaf(-tb, tb, 1.f)),
                          tc::f2_to_h2(__uint_as_float(dz[i]), __uint_as_float(dz[i + 1])),
                          res_pair<MD::Z2>(d1, c, h1lo));
      }
    }
    st_pairs(h2 + off(k8), hv[0], hv[1], hv[2], hv[3]);
    if (TANGENT) st_pairs(h2t + off(k8), dv[0], dv[1], dv[2], dv[3]);
  }
}

// Row geometry for layer 0 alone: s~ = (s(r) - mean) / std (the fast-reciprocal
// form of row_geom_mixed).
__device__ __forceinline__ float row_stilde(float4 rb, float rcut, float inv_std, float mean) {
  RowGeom g;
  row_geom_mixed(make_float3(rb.x, rb.y, rb.z), rcut, g);
  return (g.s - mean) * inv_std;
}

// ---------------------------------------------------------------- embedding forward (FP16 tcgen05)
// Per block of 8 centre atoms of type ti: neighbour rows with s(r) != 0 are
// compacted block-wide into 128-row tiles.  Two threads serve each row (TMEM
// lane): warps w and w + 4 share lane quarter w % 4 and split the columns of
// every layer (HalfSplit), so 16 warps per SM hide the latencies of the three
// MMA round trips per tile:
//   layer 0 (1 -> E0) on CUDA cores, h0 -> A0 (fp16, ones column at E0)
//   D  = A0 . [W1; b1]   (tcgen05, 128 x N1)   -> h1 = tanh(D) + rep(h0) -> A1
//   D  = A1 . [W2; b2]   (tcgen05, 128 x N2)   -> h2 = tanh(D) + rep(h1) -> H2
//   D3 += Rblk . H2 (tcgen05, M = 8 slots x 16 channels, K = 128 rows)
// where Rblk holds each row's env row R~ in its atom's 16-lane slot (zero
// elsewhere), so D3 accumulates T_a = sum_rows R~^T h2 for the 8 atoms in
// TMEM across all tiles of both neighbour types.  The block epilogue writes
// T / Nnbrs (FP32) and the descriptor G (FP16, dpmodel.py:74-78).  Only the
// current neighbour type's net is resident (2 CTAs per SM).
constexpr int kRblkBytes = 128 * 128 * 2;
constexpr int kFwdThreads = 256;
constexpr int kFwdCpt = 2;  // compaction candidates per thread, forward
constexpr int kRowCapFwd = 128 + kFwdThreads * kFwdCpt;  // the carry (< 128) + one compaction round

template <int E0, int E1, int E2>
__global__ void __launch_bounds__(kFwdThreads, 2) k_mix_embed_fwd(DevModel M, SysDesc D, int wave,
                                                                  const float4 *__restrict__ posS,
                                                                  const float *__restrict__ box,
                                                                  const int32_t *__restrict__ nbrs,
                                                                  float *__restrict__ Tout,
                                                                  __half *__restrict__ Gout,
                                                                  const float4 *__restrict__ rows_g,
                                                                  const int *__restrict__ rcnt,
                                                                  int *__restrict__ err) {
  using MD = MixDims<E0, E1, E2>;
  using SP = HalfSplit<E0, E1, E2>;
  extern __shared__ __align__(128) char smem[];
  char *netb = smem;
  float *small = reinterpret_cast<float *>(netb + round1k(MD::NETB));
  char *opa = reinterpret_cast<char *>(small) + round1k(MD::NSMALL * 4);
  char *rblk = opa + round1k(MD::OPA);
  float4 *rowbuf = reinterpret_cast<float4 *>(rblk + kRblkBytes);
  __shared__ int wcnt[kFwdThreads / 32];
  __shared__ float3 ri_s[kBlkAtoms];
  __shared__ __align__(8) uint64_t mbar;
  __shared__ uint32_t tbase_s;
  const int tid = threadIdx.x, warp = tc::warp_index();
  const int row = tid & 127, half = tid >> 7;

  for (int e = tid; e < kRblkBytes / 16; e += kFwdThreads) reinterpret_cast<uint4 *>(rblk)[e] = make_uint4(0, 0, 0, 0);
  if (tid == 0) tc::mbar_init(&mbar, 1);
  if (warp == 0) tc::tmem_alloc(&tbase_s, 256);
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tbase = tbase_s;
  const uint32_t tD = tbase, tD3 = tbase + 128, lane_off = (uint32_t)((warp & 3) * 32) << 16;
  uint32_t ph = 0;
  bool ok = true;

  const int nblk = blocks_total(D, kBlkAtoms);
  const uint32_t idesc1 = tc::idesc_f16(128, MD::N1, 0, 0);
  const uint32_t idesc2 = tc::idesc_f16(128, MD::N2, 0, 0);
  const uint32_t idesc3 = tc::idesc_f16(128, MD::N2, 1, 1);
  const uint32_t opa_u = tc::smem_u32(opa), rblk_u = tc::smem_u32(rblk);
  const uint32_t w1_u = tc::smem_u32(netb), w2_u = w1_u + MD::W1B;
  auto h2off = [row](int k8) { return tc::mnmajor_off(row, k8, MD::N2); };
  int loaded_net = -1;

  for (int blk = blockIdx.x; blk < nblk && ok; blk += gridDim.x) {
    const BlkPos bp = block_pos(D, kBlkAtoms, blk);
    const int ti = bp.ti, f = bp.f, nb = bp.nb;
    const size_t g0 = bp.g0;
    const size_t frame_base = (size_t)f * D.N;
    const float inv_std = M.inv_std[ti], mean = M.mean[ti];
    if (blk + (int)gridDim.x < nblk) {  // the next block's neighbour rows
      const BlkPos bn = block_pos(D, kBlkAtoms, blk + gridDim.x);
      if (rows_g != nullptr && D.S <= kRowStoreCap)
        prefetch_range_l2(rows_g + bn.g0 * kRowStoreCap, (size_t)bn.nb * D.S * 16);
      else prefetch_range_l2(nbrs + bn.g0 * D.S, (size_t)bn.nb * D.S * 4);
    }
    const int bs = box_slot(D, g0, f);  // the block's 8 atoms share one frame
    const float3 L = make_float3(box[bs * 3], box[bs * 3 + 1], box[bs * 3 + 2]);
    const int3 ni = image_range(L, M.rcut);
    const int nim = (2 * ni.x + 1) * (2 * ni.y + 1) * (2 * ni.z + 1);
    const bool stream = row_store_covers(D, rows_g, nim);  // the block's rows are in the store
    if (stream && blk == (int)blockIdx.x) prefetch_range_l2(rows_g + g0 * kRowStoreCap, (size_t)nb * D.S * 16);
    if (tid < nb) {
      const float4 q = posS[g0 + tid];
      ri_s[tid] = make_float3(q.x, q.y, q.z);
    }
    __syncthreads();
    int ntile = 0;
    bool pending = false;
    int my_slot = -1;
    int rowstart = 0, rowcount = 0;
    // The neighbour types' order rotates from one wave of `wave` blocks of a centre
    // type to the next, so that the resident net mostly carries over; it depends on
    // the block alone, so T's rounding does not depend on the launch.
    const int local = blk - bp.first, turn = local / min(blocks_of_type(D, ti, kBlkAtoms), wave);
    const int tj0 = turn * (D.ntypes - 1) % D.ntypes;
    for (int tt = 0; tt < D.ntypes && ok; ++tt) {
      const int tj = (tj0 + tt) % D.ntypes;
      const int sel = D.sel[tj];
      const int per_atom = sel * nim, total = nb * per_atom;
      const float *sm = small;
      const int knet = ti * M.ntypes + tj;
      const float4 *rsrc = stream ? rows_g + g0 * kRowStoreCap + (size_t)nb * D.col[tj] : nullptr;
      const int nsrc = stream ? rcnt[g0 * M.ntypes + tj] : total;  // stored rows, or candidates
      constexpr int step = kFwdThreads * kFwdCpt;  // candidates, or stored rows, per round
      for (int base = 0; base < nsrc + step && ok; base += step) {
        const bool flush = base >= nsrc;
        if (!flush) {
          if (stream)
            mix_stream_round<kFwdCpt>(rsrc, base, nsrc, rowbuf, rowstart, rowcount);
          else
            mix_compact_round<kFwdCpt>(D, M, tj, base, total, per_atom, nim, ni, L, g0, frame_base, ri_s, posS,
                                       nbrs, rowbuf, wcnt, rowstart, rowcount);
        }
        while (rowcount - rowstart >= 128 || (flush && rowcount > rowstart)) {
          const int nrows = min(rowcount - rowstart, 128);
          if (pending) {  // previous contraction done: operands free, clear its Rblk entries
            MIX_WAIT();
            pending = false;
            if (!ok) break;
            if (half == 0 && my_slot >= 0) {
              const uint32_t o = tc::mnmajor_off(row, 16 * my_slot, 128);
              *reinterpret_cast<uint4 *>(rblk + o) = make_uint4(0, 0, 0, 0);
              *reinterpret_cast<uint4 *>(rblk + o + 128) = make_uint4(0, 0, 0, 0);
            }
          }
          if (loaded_net != knet) {  // resident net of this neighbour type
            __syncthreads();
            mix_load_net<E0, E1, E2>(M, knet, netb, small);
            loaded_net = knet;
          }
          const bool act = row < nrows;
          const float4 rv = act ? rowbuf[rowstart + row] : make_float4(100.f, 100.f, 100.f, 0.f);
          const int slot = act ? (__float_as_int(rv.w) & 7) : -1;
          RowGeom gm;
          float st, R[10];
          mix_row_env(rv, M.rcut, inv_std, mean, gm, st, R);
          tc::cp_async_wait<0>();
          __syncthreads();  // net image visible; rowbuf read by every thread
          __half2 h0[SP::NP0], h1[SP::NP1];
          if (half == 0) emb_layer0<E0, E1, E2, 0, false>(st, sm, row, opa, nullptr, h0, h0);
          else emb_layer0<E0, E1, E2, 1, false>(st, sm, row, opa, nullptr, h0, h0);
          my_slot = slot;
          if (half == 0 && act) {
            const uint32_t o = tc::mnmajor_off(row, 16 * slot, 128);
            st_pairs(rblk + o, tc::f2_to_h2(R[0], R[1]), tc::f2_to_h2(R[2], R[3]), tc::f2_to_h2(R[4], R[5]),
                     tc::f2_to_h2(R[6], R[7]));
            *reinterpret_cast<uint4 *>(rblk + o + 128) = make_uint4(tc::as_u32(tc::f2_to_h2(R[8], R[9])), 0u, 0u, 0u);
          }
          tc::fence_proxy_async();
          tc::fence_before_sync();
          __syncthreads();
          if (warp == 0 && tc::elect_one()) {
            tc::fence_after_sync();
#pragma unroll
            for (int ks = 0; ks < MD::K1 / 16; ++ks)
              tc::mma_f16kind(tD, tc::make_desc(opa_u + tc::kmajor_off(0, 16 * ks, MD::K1), 128, (MD::K1 / 8) * 128),
                           tc::make_desc(w1_u + tc::kmajor_off(0, 16 * ks, MD::K1), 128, (MD::K1 / 8) * 128),
                           idesc1, ks > 0);
            tc::commit(&mbar);
          }
          MIX_WAIT();
          if (!ok) break;
          if (half == 0) emb_epi1<E0, E1, E2, 0, false>(tD + lane_off, 0, row, opa, nullptr, h0, h0, h1, h1);
          else emb_epi1<E0, E1, E2, 1, false>(tD + lane_off, 0, row, opa, nullptr, h0, h0, h1, h1);
          tc::fence_proxy_async();
          tc::fence_before_sync();
          __syncthreads();
          if (warp == 0 && tc::elect_one()) {
            tc::fence_after_sync();
#pragma unroll
            for (int ks = 0; ks < MD::K2 / 16; ++ks)
              tc::mma_f16kind(tD, tc::make_desc(opa_u + tc::kmajor_off(0, 16 * ks, MD::K2), 128, (MD::K2 / 8) * 128),
                           tc::make_desc(w2_u + tc::kmajor_off(0, 16 * ks, MD::K2), 128, (MD::K2 / 8) * 128),
                           idesc2, ks > 0);
            tc::commit(&mbar);
          }
          MIX_WAIT();
          if (!ok) break;
          if (half == 0) emb_epi2<E0, E1, E2, 0, false>(tD + lane_off, 0, opa, nullptr, h2off, h1, h1);
          else emb_epi2<E0, E1, E2, 1, false>(tD + lane_off, 0, opa, nullptr, h2off, h1, h1);
          tc::fence_proxy_async();
          tc::fence_before_sync();
          __syncthreads();
          if (warp == 0 && tc::elect_one()) {
            tc::fence_after_sync();
#pragma unroll
            for (int ks = 0; ks < 8; ++ks)
              tc::mma_f16kind(tD3, tc::make_desc(rblk_u + tc::mnmajor_off(16 * ks, 0, 128), (128 / 8) * 128, 128),
                           tc::make_desc(opa_u + tc::mnmajor_off(16 * ks, 0, MD::N2), (MD::N2 / 8) * 128, 128),
                           idesc3, (ntile > 0 || ks > 0) ? 1u : 0u);
            tc::commit(&mbar);
          }
          pending = true;
          ++ntile;
          rowstart += nrows;
        }
      }
    }
    if (!ok) break;
    if (pending) {
      MIX_WAIT();
      pending = false;
      if (!ok) break;
      if (half == 0 && my_slot >= 0) {
        const uint32_t o = tc::mnmajor_off(row, 16 * my_slot, 128);
        *reinterpret_cast<uint4 *>(rblk + o) = make_uint4(0, 0, 0, 0);
        *reinterpret_cast<uint4 *>(rblk + o + 128) = make_uint4(0, 0, 0, 0);
      }
    }
    // ---- block epilogue: T (FP32) and G (FP16) from the TMEM accumulators
    __syncthreads();
    float *Xs = reinterpret_cast<float *>(rblk);  // T staging [slot][c][w], 8 x 10 x E2 floats
    {
      const int slot = row >> 4, c = row & 15;
      constexpr int NG = MD::N2 / 16, NG0 = (NG + 1) / 2;  // column groups of half 0
      const int q0 = half ? NG0 : 0, q1 = half ? NG : NG0;
      for (int q = q0; q < q1; q += 2) {
        const int c0 = 16 * q;
        const bool two = q + 1 < q1;  // warp-uniform
        uint32_t r[2][16];
        if (ntile > 0) {
          tc::tmem_ld16_issue(tD3 + lane_off + c0, r[0]);
          if (two) tc::tmem_ld16_issue(tD3 + lane_off + c0 + 16, r[1]);
          tc::tmem_wait();
        } else {
#pragma unroll
          for (int i = 0; i < 16; ++i) r[0][i] = r[1][i] = 0u;
        }
        if (slot < nb && c < 10) {
#pragma unroll
          for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int i = 0; i < 16; ++i) {
              const int w = c0 + 16 * h + i;
              if ((h == 0 || two) && w < E2) Xs[(slot * 10 + c) * E2 + w] = __uint_as_float(r[h][i]) * M.inv_nnbrs;
            }
        }
      }
    }
    tc::fence_before_sync();
    __syncthreads();
    {  // the block's T rows are contiguous in Tout and in Xs: coalesced copy
      const int n4 = nb * 10 * E2 / 4;
      float4 *dst = reinterpret_cast<float4 *>(Tout + g0 * 10 * E2);
      const float4 *src = reinterpret_cast<const float4 *>(Xs);
      for (int e = tid; e < n4; e += kFwdThreads) dst[e] = src[e];
    }
    // G[a][w] = sum_c Q[c][a] X[c][w] with X = T + Tbias on channel 0
    // (dpmodel.py:74-78): Q of every slot is staged once (zero for a >= A),
    // then a thread owns (slot, column pair) items, keeps X[.][w], X[.][w+1]
    // in registers and reads Q as warp-wide broadcasts.
    const int A = M.A;
    float *Qs = Xs + kBlkAtoms * 10 * E2;  // [slot][c][16], past Rblk into the (idle) row buffer
    for (int e = tid; e < kBlkAtoms * 160; e += kFwdThreads) {
      const int slot = e / 160, c = (e >> 4) % 10, aa = e & 15;
      float q = 0.f;
      if (slot < nb && aa < A) {
        const float *X = Xs + slot * 10 * E2;
        if (c < 4) {
          q = X[c * E2 + aa] + (c == 0 ? M.tbias[aa] : 0.f);
        } else {
          const float y1 = X[E2 + A + aa], y2 = X[2 * E2 + A + aa], y3 = X[3 * E2 + A + aa];
          const float b6[6] = {y1 * y1, y2 * y2, y3 * y3, kSqrt2 * y1 * y3, kSqrt2 * y2 * y1, kSqrt2 * y3 * y2};
          q = b6[c - 4] + X[c * E2 + A + aa];
        }
      }
      Qs[e] = q;
    }
    __syncthreads();
    constexpr int WP2 = (E2 / 2 + 31) / 32 * 32;  // column pairs per slot, whole warps
    for (int pr = tid; pr < nb * WP2; pr += kFwdThreads) {
      const int slot = pr / WP2, w = 2 * (pr - slot * WP2);
      if (w < E2) {
        float xa[10], xb[10];
#pragma unroll
        for (int c = 0; c < 10; ++c) {
          const float2 v = *reinterpret_cast<const float2 *>(Xs + (slot * 10 + c) * E2 + w);
          xa[c] = v.x;
          xb[c] = v.y;
        }
        xa[0] += M.tbias[w];
        xb[0] += M.tbias[w + 1];
        const float *Q = Qs + slot * 160;
        __half2 *Gs = reinterpret_cast<__half2 *>(Gout + (g0 + slot) * (size_t)A * E2 + w);
        for (int aa = 0; aa < A; ++aa) {
          float va = 0.f, vb = 0.f;
#pragma unroll
          for (int c = 0; c < 10; ++c) {
            const float qv = Q[c * 16 + aa];
            va = fmaf(qv, xa[c], va);
            vb = fmaf(qv, xb[c], vb);
          }
          Gs[aa * (E2 / 2)] = __floats2half2_rn(va, vb);  // no saturation: |G| > 65504 -> inf -> NaN energy
        }
      }
    }
    __syncthreads();
    for (int e = tid; e < kRblkBytes / 16; e += kFwdThreads) reinterpret_cast<uint4 *>(rblk)[e] = make_uint4(0, 0, 0, 0);
    __syncthreads();
  }
  if (!ok) {
    if (tid == 0) atomicOr(err, 1);
    tc::mbar_wait(&mbar, ph);
  }
  tc::cp_async_wait<0>();
  tc::fence_before_sync();
  __syncthreads();
  if (warp == 0) tc::tmem_dealloc(tbase, 256);
}

template <int E0, int E1, int E2>
size_t mix_fwd_smem() {
  using MD = MixDims<E0, E1, E2>;
  return (size_t)round1k(MD::NETB) + round1k(MD::NSMALL * 4) + round1k(MD::OPA) + kRblkBytes + kRowCapFwd * 16;
}

static int num_sms() {
  int dev = 0, nsm = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  return nsm;
}

template <int E0, int E1, int E2>
int launch_mix_embed_fwd(const DevModel &M, const SysDesc &D, const float4 *posS,
                         const float *box, const int32_t *nbrs, float *T, __half *G, const float4 *rows_g,
                         const int *rcnt, int *err, cudaStream_t st) {
  const int nblk = blocks_total(D, kBlkAtoms);
  if (nblk == 0) return DPB_OK;
  const size_t smem = mix_fwd_smem<E0, E1, E2>();
  DPB_CUDA_TRY(cudaFuncSetAttribute(k_mix_embed_fwd<E0, E1, E2>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)smem));
  const int wave = 2 * num_sms(), grid = nblk < wave ? nblk : wave;
  k_mix_embed_fwd<E0, E1, E2><<<grid, kFwdThreads, smem, st>>>(M, D, wave, posS, box, nbrs, T, G, rows_g, rcnt,
                                                                err);
  count_launch();
  DPB_LAUNCH_CHECK();
  return DPB_OK;
}

// ---------------------------------------------------------------- dE/dT (warp per atom, warp-level MMA)
// Adjoint of the descriptor (dpmodel.py:74-78): G[a][w] = sum_c Q[c][a] X[c][w]
// with X = T + Tbias on channel 0 and Q[c][a] = X[c][a] (c < 4), the y_c
// products of X[1..3][A + a] plus X[c][A + a] (c >= 4).  From dE/dG (FP16
// times fit_dgsc, from the fitting chain) and T, per atom
//   dQ[c][a] = sum_w X[c][w] dG[a][w]       (16 x 16 x N2 on mma.sync)
//   dX[c][w] = sum_a Q[c][a] dG[a][w]       (16 x N2 x 16 on mma.sync)
//            + the Q -> X terms at w < 2A   (FP32)
// and dE/dT / Nnbrs leaves as FP16 rows [atom][c][w] (w padded to N2 with
// zeros), the B operand rows of the tensor-core adjoint, each atom's rows
// scaled by the power of two 2^k that puts their largest magnitude in
// [2^13, 2^14); dTs[atom] = 2^-k / fit_dgsc undoes both scales.  X and Q
// enter the FP16 products as their rounded value plus the rounded remainder
// (hi + lo, about 22 significant bits), dE/dG is FP16 already, and the
// products accumulate in FP32.  Each warp stages its atom in shared memory
// (X hi / lo and the dE/dG rows at a padded row stride, so the ldmatrix
// reads of eight rows hit distinct banks).
template <int E2, int N2>
struct DtCfg {
  static constexpr int XS = N2 + 8;       // row stride (halves) of X and dE/dG
  static constexpr int QS = 24;           // row stride (halves) of Q
  static constexpr int XB = 16 * XS * 2;  // one 16-row FP16 tile
  static constexpr int QB = 16 * QS * 2;
  static constexpr int WARP_BYTES = 3 * XB + 2 * QB + 16 * 16 * 4 + 48 * 4;
  static_assert(XB % 16 == 0 && WARP_BYTES % 16 == 0, "16-byte aligned tiles");
};

template <int E2, int N2, int W>
__global__ void __launch_bounds__(32 * W) k_mix_dT(DevModel M, int NF, const float *__restrict__ Tin,
                                                const __half *__restrict__ dG,
                                                __half *__restrict__ dTh, float *__restrict__ dTs) {
  using C = DtCfg<E2, N2>;
  constexpr int XS = C::XS, QS = C::QS;
  static_assert(E2 % 4 == 0 && E2 >= 32 && N2 % 16 == 0 && N2 >= E2 && N2 - E2 < 16, "dE/dT tile widths");
  extern __shared__ __align__(16) char dt_smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const size_t stride = (size_t)gridDim.x * W;  // warp-strided atoms
  size_t g = (size_t)blockIdx.x * W + warp;
  if (g >= (size_t)NF) return;
  char *wb = dt_smem + warp * C::WARP_BYTES;
  __half *Xh = reinterpret_cast<__half *>(wb), *Xl = Xh + 16 * XS, *Dg = Xl + 16 * XS;
  __half *Qh = Dg + 16 * XS, *Ql = Qh + 16 * QS;
  float *dQs = reinterpret_cast<float *>(Ql + 16 * QS);  // [c][a], 16 x 16
  float *ys = dQs + 256;                                 // [k][a]: y_{k+1}[a] = X[k + 1][A + a]
  const int A = M.A;                                     // 1..16 (2A <= 32 <= E2)
  // ---- zero padding of the tiles, once (the atoms' stages never write it)
  const uint2 z2 = make_uint2(0u, 0u);
  for (int e = lane; e < 6 * (XS / 4); e += 32) {  // X rows 10..15
    reinterpret_cast<uint2 *>(Xh + 10 * XS)[e] = z2;
    reinterpret_cast<uint2 *>(Xl + 10 * XS)[e] = z2;
  }
  for (int e = lane; e < (16 - A) * (XS / 4); e += 32) reinterpret_cast<uint2 *>(Dg + A * XS)[e] = z2;  // rows a >= A
  if constexpr (N2 > E2) {  // columns [E2, N2) of the live rows
    constexpr int PW = (N2 - E2) / 4;
    for (int e = lane; e < 10 * PW; e += 32) {
      const int r = e / PW, o = E2 + 4 * (e - r * PW);
      *reinterpret_cast<uint2 *>(Xh + r * XS + o) = z2;
      *reinterpret_cast<uint2 *>(Xl + r * XS + o) = z2;
    }
    for (int e = lane; e < A * PW; e += 32) {
      const int r = e / PW, o = E2 + 4 * (e - r * PW);
      *reinterpret_cast<uint2 *>(Dg + r * XS + o) = z2;
    }
  }
  // ---- an atom's global inputs in registers: T rows (float4), dE/dG rows
  // (4 halves), the Q inputs; the next atom's are loaded right after this
  // atom's are staged, so they arrive while this atom's products run
  constexpr int N4 = 10 * E2 / 4, K4 = (N4 + 31) / 32;
  constexpr int P4 = E2 / 4, NP = 16 * P4, KP = (NP + 31) / 32;
  const int aq = lane & 15;
  const bool qlane = lane < 16 && aq < A;
  float4 tv[K4];
  uint2 dv[KP];
  float xr[4], xt[10];
  auto load = [&](size_t ga) {
    const float *Tg = Tin + ga * 10 * E2;
#pragma unroll
    for (int k = 0; k < K4; ++k) {
      const int e4 = lane + 32 * k;
      tv[k] = e4 < N4 ? reinterpret_cast<const float4 *>(Tg)[e4] : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    const uint2 *Dg8 = reinterpret_cast<const uint2 *>(dG + ga * (size_t)A * E2);
#pragma unroll
    for (int k = 0; k < KP; ++k) {
      const int p = lane + 32 * k, a = p / P4;
      dv[k] = (p < NP && a < A) ? Dg8[p] : make_uint2(0u, 0u);
    }
#pragma unroll
    for (int c = 0; c < 4; ++c) xr[c] = qlane ? Tg[c * E2 + aq] : 0.f;
#pragma unroll
    for (int c = 1; c < 10; ++c) xt[c] = qlane ? Tg[c * E2 + A + aq] : 0.f;
  };
  load(g);
  for (; g < (size_t)NF; g += stride) {
#pragma unroll
  for (int k = 0; k < K4; ++k) {
    const int e4 = lane + 32 * k;
    if (e4 < N4) {
      const int e = 4 * e4, c = e / E2, w = e - c * E2;
      float x[4] = {tv[k].x, tv[k].y, tv[k].z, tv[k].w};
      if (c == 0) {
#pragma unroll
        for (int i = 0; i < 4; ++i) x[i] += M.tbias[w + i];
      }
      __half h[4], l[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        h[i] = __float2half_rn(x[i]);
        l[i] = __float2half_rn(x[i] - __half2float(h[i]));
      }
      *reinterpret_cast<uint2 *>(Xh + c * XS + w) =
          make_uint2(tc::as_u32(__halves2half2(h[0], h[1])), tc::as_u32(__halves2half2(h[2], h[3])));
      *reinterpret_cast<uint2 *>(Xl + c * XS + w) =
          make_uint2(tc::as_u32(__halves2half2(l[0], l[1])), tc::as_u32(__halves2half2(l[2], l[3])));
    }
  }
#pragma unroll
  for (int k = 0; k < KP; ++k) {
    const int p = lane + 32 * k, a = p / P4;
    if (p < NP && a < A) *reinterpret_cast<uint2 *>(Dg + a * XS + 4 * (p - a * P4)) = dv[k];
  }
  if (lane < 16) {  // Q[c][a] of column a = lane (zero for a >= A and rows c >= 10), and y
    float q[10];
    const float y1 = xt[1], y2 = xt[2], y3 = xt[3];
    q[0] = xr[0] + (qlane ? M.tbias[aq] : 0.f);
    q[1] = xr[1]; q[2] = xr[2]; q[3] = xr[3];
    const float b6[6] = {y1 * y1, y2 * y2, y3 * y3, kSqrt2 * y1 * y3, kSqrt2 * y2 * y1, kSqrt2 * y3 * y2};
#pragma unroll
    for (int m = 0; m < 6; ++m) q[4 + m] = b6[m] + xt[4 + m];
#pragma unroll
    for (int c = 0; c < 16; ++c) {
      const float v = (c < 10 && qlane) ? fminf(fmaxf(q[c < 10 ? c : 0], -65504.f), 65504.f) : 0.f;
      const __half h = __float2half_rn(v);
      Qh[c * QS + aq] = h;
      Ql[c * QS + aq] = __float2half_rn(v - __half2float(h));
    }
    ys[aq] = y1;
    ys[16 + aq] = y2;
    ys[32 + aq] = y3;
  }
  if (g + stride < (size_t)NF) load(g + stride);
  __syncwarp();
  // ---- dQ = X . dE/dG^T: M = c, N = a (two tiles of 8), K = w
  const int g8 = lane >> 2, q4 = lane & 3, mi = lane >> 3, ri = lane & 7;
  float acc[2][4];
#pragma unroll
  for (int n = 0; n < 2; ++n)
#pragma unroll
    for (int i = 0; i < 4; ++i) acc[n][i] = 0.f;
#pragma unroll
  for (int kt = 0; kt < N2 / 16; ++kt) {
    uint32_t ah[4], al[4];
    const int arow = (ri + 8 * (mi & 1)) * XS + 16 * kt + 8 * (mi >> 1);
    tc::ldmatrix_x4(ah, Xh + arow);
    tc::ldmatrix_x4(al, Xl + arow);
#pragma unroll
    for (int n = 0; n < 2; ++n) {
      uint32_t b0, b1;
      tc::ldmatrix_x2(b0, b1, Dg + (8 * n + ri) * XS + 16 * kt + 8 * (mi & 1));
      tc::mma_16816(acc[n], ah, b0, b1);
      tc::mma_16816(acc[n], al, b0, b1);
    }
  }
#pragma unroll
  for (int n = 0; n < 2; ++n) {
    const int a = 8 * n + 2 * q4;
    dQs[g8 * 16 + a] = acc[n][0];
    dQs[g8 * 16 + a + 1] = acc[n][1];
    dQs[(g8 + 8) * 16 + a] = acc[n][2];
    dQs[(g8 + 8) * 16 + a + 1] = acc[n][3];
  }
  // ---- dX = Q . dE/dG: M = c, N = w (tiles of 8), K = a
  uint32_t qh[4], ql[4];
  {
    const int qrow = (ri + 8 * (mi & 1)) * QS + 8 * (mi >> 1);
    tc::ldmatrix_x4(qh, Qh + qrow);
    tc::ldmatrix_x4(ql, Ql + qrow);
  }
  float o[N2 / 8][4];
#pragma unroll
  for (int nt = 0; nt < N2 / 8; ++nt) {
    uint32_t b0, b1;
    tc::ldmatrix_x2_trans(b0, b1, Dg + (ri + 8 * (mi & 1)) * XS + 8 * nt);
#pragma unroll
    for (int i = 0; i < 4; ++i) o[nt][i] = 0.f;
    tc::mma_16816(o[nt], qh, b0, b1);
    tc::mma_16816(o[nt], ql, b0, b1);
  }
  __syncwarp();  // dQs of every lane
  // ---- Q -> X terms (w < 2A), 1 / Nnbrs, zero past E2 and for rows c >= 10
  float amax = 0.f;
#pragma unroll
  for (int nt = 0; nt < N2 / 8; ++nt)
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int c = g8 + 8 * (i >> 1), w = 8 * nt + 2 * q4 + (i & 1);
      float x = o[nt][i];
      if (8 * nt < 32 && c < 10) {
        if (w < A) {
          if (c < 4) x += dQs[c * 16 + w];
        } else if (w < 2 * A) {
          const int aa = w - A;
          if (c >= 4) {
            x += dQs[c * 16 + aa];
          } else if (c >= 1) {
            const float y1 = ys[aa], y2 = ys[16 + aa], y3 = ys[32 + aa];
            const float d0 = dQs[64 + aa], d1 = dQs[80 + aa], d2 = dQs[96 + aa], d3 = dQs[112 + aa],
                        d4 = dQs[128 + aa], d5 = dQs[144 + aa];
            if (c == 1) x += 2.f * y1 * d0 + kSqrt2 * y3 * d3 + kSqrt2 * y2 * d4;
            if (c == 2) x += 2.f * y2 * d1 + kSqrt2 * y1 * d4 + kSqrt2 * y3 * d5;
            if (c == 3) x += 2.f * y3 * d2 + kSqrt2 * y1 * d3 + kSqrt2 * y2 * d5;
          }
        }
      }
      x = (c < 10 && w < E2) ? x * M.inv_nnbrs : 0.f;
      o[nt][i] = x;
      amax = fmaxf(amax, fabsf(x));
    }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, off));
  // amax = m 2^e with m in [0.5, 1): scale 2^(14 - e) puts it in [2^13, 2^14)
  int e = 0;
  const bool fin = amax > 0.f && amax < INFINITY;
  if (fin) frexpf(amax, &e);
  const int k = fin ? 14 - e : 0;
  const float scale = ldexpf(1.f, k);
  if (lane == 0) dTs[g] = ldexpf(1.f, -k) / M.fit_dgsc;
  __half *out = dTh + g * 10 * N2;
#pragma unroll
  for (int nt = 0; nt < N2 / 8; ++nt) {
    const int w = 8 * nt + 2 * q4;
    *reinterpret_cast<__half2 *>(out + g8 * N2 + w) = tc::f2_to_h2(o[nt][0] * scale, o[nt][1] * scale);
    if (g8 + 8 < 10)
      *reinterpret_cast<__half2 *>(out + (g8 + 8) * N2 + w) = tc::f2_to_h2(o[nt][2] * scale, o[nt][3] * scale);
  }
  __syncwarp();  // every lane is done with this atom's tiles before the next stage
  }
}

// ---------------------------------------------------------------- embedding adjoint (FP16 tcgen05)
// Per block of 8 centre atoms: the B tile DTB holds the atoms' dE/dT rows
// (FP16, each atom's rows scaled by a power of two, k_mix_dT) as rows
// n = 16 slot + c (c < 10; rows 10..15 of a slot zero), K = N2.  The rows are
// recomputed with their tangent along s~ (forward mode), two threads per row
// as in the forward kernel: [h0, dh0] -> tcgen05 -> [h1, dh1] -> tcgen05 ->
// [h2, dh2], then U = H2 . DTB and V = dH2 . DTB on the tensor cores over the
// slots the tile's rows belong to only (N = 16 x the tile's slot count; rows
// are sorted by slot); a row reads its slot's 16 columns: u = dE/dR~ and
// dE/ds~ = R~ . v.  The FP32 row adjoint gives dE/dx (unscaled by the atom's
// factor); half 0 scatters it as the neighbour's force and sums the virial,
// half 1 reduces the centre atoms' forces.  One resident net, 2 CTAs per SM.
constexpr int kBwdThreads = 256;
constexpr int kBwdCpt = 1;  // compaction candidates per thread, adjoint
constexpr int kRowCapBwd = 128 + kBwdThreads * kBwdCpt;
constexpr int kDtbRows = 16 * kBlkAtoms;  // DTB rows: 16 per atom slot

template <int E0, int E1, int E2>
__global__ void __launch_bounds__(kBwdThreads, 2) k_mix_embed_bwd(DevModel M, SysDesc D,
                                                                  const float4 *__restrict__ posS,
                                                                  const float *__restrict__ box,
                                                                  const int32_t *__restrict__ nbrs,
                                                                  const __half *__restrict__ dTh,
                                                                  const float *__restrict__ dTs,
                                                                  const float4 *__restrict__ rows_g,
                                                                  const int *__restrict__ rcnt,
                                                                  ForceSum *__restrict__ F4,
                                                                  double *__restrict__ virial,
                                                                  int *__restrict__ err) {
  using MD = MixDims<E0, E1, E2>;
  using SP = HalfSplit<E0, E1, E2>;
  constexpr int DTB_BYTES = kDtbRows * MD::N2 * 2;
  extern __shared__ __align__(128) char smem[];
  char *netb = smem;
  float *small = reinterpret_cast<float *>(netb + round1k(MD::NETB));
  char *dtb = reinterpret_cast<char *>(small) + round1k(MD::NSMALL * 4);
  char *opb = dtb + round1k(DTB_BYTES);
  float4 *rowbuf = reinterpret_cast<float4 *>(opb + round1k(2 * MD::OPA));
  __shared__ int wcnt[kBwdThreads / 32];
  __shared__ float3 ri_s[kBlkAtoms];
  __shared__ int src_s[kBlkAtoms];  // user index of each centre
  __shared__ float sc_s[kBlkAtoms];
  __shared__ double vir_s[9];
  __shared__ __align__(8) uint64_t mbar;
  __shared__ uint32_t tbase_s;
  const int tid = threadIdx.x, warp = tc::warp_index(), lane = tid & 31;
  const int row = tid & 127, half = tid >> 7;

  if (tid < 9) vir_s[tid] = 0.0;
  if (tid == 0) tc::mbar_init(&mbar, 1);
  if (warp == 0) tc::tmem_alloc(&tbase_s, 256);
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tbase = tbase_s, lane_off = (uint32_t)((warp & 3) * 32) << 16;
  uint32_t ph = 0;
  bool ok = true;
  float vir[9];
#pragma unroll
  for (int k = 0; k < 9; ++k) vir[k] = 0.f;
  // the virial goes to the frame of the blocks processed; a CTA that moves on
  // to a block of another frame (packed batches) flushes its sum first
  int vframe = -1;
  auto flush_virial = [&]() {
#pragma unroll
    for (int k = 0; k < 9; ++k) {
      const float s = warp_sum(vir[k]);
      if (lane == 0 && s != 0.f) atomicAdd(&vir_s[k], (double)s);
      vir[k] = 0.f;
    }
    __syncthreads();
    if (tid < 9) {
      atomicAdd(&virial[vframe * 9 + tid], vir_s[tid]);
      vir_s[tid] = 0.0;
    }
    __syncthreads();
  };

  const int nblk = blocks_total(D, kBlkAtoms);
  const uint32_t idesc1 = tc::idesc_f16(128, MD::N1, 0, 0);
  const uint32_t idesc2 = tc::idesc_f16(128, MD::N2, 0, 0);
  const uint32_t opb_u = tc::smem_u32(opb), dtb_u = tc::smem_u32(dtb);
  const uint32_t w1_u = tc::smem_u32(netb), w2_u = w1_u + MD::W1B;
  // operand offsets in opb: each layer's value operand at 0, its tangent at OPA
  constexpr uint32_t kTan = MD::OPA;
  auto h2off = [row](int k8) { return tc::kmajor_off(row, k8, MD::N2); };
  int loaded_net = -1;

  for (int blk = blockIdx.x; blk < nblk && ok; blk += gridDim.x) {
    const BlkPos bp = block_pos(D, kBlkAtoms, blk);
    const int ti = bp.ti, f = bp.f, nb = bp.nb;
    const size_t g0 = bp.g0;
    const size_t frame_base = (size_t)f * D.N;
    const float inv_std = M.inv_std[ti], mean = M.mean[ti];
    if (blk + (int)gridDim.x < nblk) {  // the next block's neighbour rows and dE/dT rows
      const BlkPos bn = block_pos(D, kBlkAtoms, blk + gridDim.x);
      if (rows_g != nullptr && D.S <= kRowStoreCap)
        prefetch_range_l2(rows_g + bn.g0 * kRowStoreCap, (size_t)bn.nb * D.S * 16);
      else prefetch_range_l2(nbrs + bn.g0 * D.S, (size_t)bn.nb * D.S * 4);
      prefetch_range_l2(dTh + bn.g0 * 10 * MD::N2, (size_t)bn.nb * 10 * MD::N2 * 2);
    }
    const int bs = box_slot(D, g0, f);  // the block's 8 atoms share one frame
    if (bs != vframe) {
      if (vframe >= 0) flush_virial();
      vframe = bs;
    }
    const float3 L = make_float3(box[bs * 3], box[bs * 3 + 1], box[bs * 3 + 2]);
    const int3 ni = image_range(L, M.rcut);
    const int nim = (2 * ni.x + 1) * (2 * ni.y + 1) * (2 * ni.z + 1);
    // the rows the forward kernel kept for this block (list mode), else compact again
    const bool stream = rows_g != nullptr && nim == 1 && D.S <= kRowStoreCap;
    if (stream && blk == (int)blockIdx.x) prefetch_range_l2(rows_g + g0 * kRowStoreCap, (size_t)nb * D.S * 16);
    if (tid < nb) {
      const float4 q = posS[g0 + tid];
      ri_s[tid] = make_float3(q.x, q.y, q.z);
      sc_s[tid] = dTs[g0 + tid];
      src_s[tid] = __float_as_int(q.w);
    }
    // ---- DTB: rows n = 16 slot + c of the 8 atoms (K-major, K = N2); zero for c >= 10 and missing atoms
    for (int e = tid; e < kDtbRows * (MD::N2 / 8); e += kBwdThreads) {
      const int n = e / (MD::N2 / 8), k8 = (e - n * (MD::N2 / 8)) * 8;
      const int slot = n >> 4, c = n & 15;
      char *dst = dtb + tc::kmajor_off(n, k8, MD::N2);
      if (slot < nb && c < 10) tc::cp_async16(dst, dTh + ((g0 + slot) * 10 + c) * MD::N2 + k8);
      else *reinterpret_cast<uint4 *>(dst) = make_uint4(0, 0, 0, 0);
    }
    tc::cp_async_commit();
    __syncthreads();
    int rowstart = 0, rowcount = 0;
    const int tj0 = (loaded_net >= 0 && loaded_net / M.ntypes == ti) ? loaded_net - ti * M.ntypes : 0;
    for (int tt = 0; tt < D.ntypes && ok; ++tt) {
      const int tj = (tj0 + tt) % D.ntypes;
      const int sel = D.sel[tj];
      const int per_atom = sel * nim, total = nb * per_atom;
      const float *sm = small;
      const int knet = ti * M.ntypes + tj;
      constexpr int kStep = kBwdThreads * kBwdCpt;
      const float4 *rsrc = stream ? rows_g + g0 * kRowStoreCap + (size_t)nb * D.col[tj] : nullptr;
      const int nsrc = stream ? rcnt[g0 * M.ntypes + tj] : total;  // stored rows, or candidates
      for (int base = 0; base < nsrc + kStep && ok; base += kStep) {
        const bool flush = base >= nsrc;
        if (!flush) {
          if (stream)
            mix_stream_round<kBwdCpt>(rsrc, base, nsrc, rowbuf, rowstart, rowcount);
          else
            mix_compact_round<kBwdCpt>(D, M, tj, base, total, per_atom, nim, ni, L, g0, frame_base, ri_s, posS,
                                       nbrs, rowbuf, wcnt, rowstart, rowcount);
        }
        while (rowcount - rowstart >= 128 || (flush && rowcount > rowstart)) {
          const int nrows = min(rowcount - rowstart, 128);
          if (loaded_net != knet) {
            __syncthreads();
            mix_load_net<E0, E1, E2>(M, knet, netb, small);
            loaded_net = knet;
          }
          const bool act = row < nrows;
          const float4 rv = act ? rowbuf[rowstart + row] : make_float4(100.f, 100.f, 100.f, 0.f);
          // rows are sorted by slot: the tile's slots are [smin, smax]
          const int smin = __float_as_int(rowbuf[rowstart].w) & 7;
          const int smax = __float_as_int(rowbuf[rowstart + nrows - 1].w) & 7;
          const float st = row_stilde(rv, M.rcut, inv_std, mean);
          tc::cp_async_wait<0>();
          __syncthreads();  // net image and DTB visible
          __half2 h1[SP::NP1], d1[SP::NP1];
          {
            __half2 h0[SP::NP0], d0[SP::NP0];
            if (half == 0) emb_layer0<E0, E1, E2, 0, true>(st, sm, row, opb, opb + kTan, h0, d0);
            else emb_layer0<E0, E1, E2, 1, true>(st, sm, row, opb, opb + kTan, h0, d0);
            tc::fence_proxy_async();
            tc::fence_before_sync();
            __syncthreads();
            if (warp == 0 && tc::elect_one()) {
              tc::fence_after_sync();
#pragma unroll
              for (int ks = 0; ks < MD::K1 / 16; ++ks) {
                const uint64_t bd = tc::make_desc(w1_u + tc::kmajor_off(0, 16 * ks, MD::K1), 128, (MD::K1 / 8) * 128);
                tc::mma_f16kind(tbase, tc::make_desc(opb_u + tc::kmajor_off(0, 16 * ks, MD::K1), 128,
                                                  (MD::K1 / 8) * 128), bd, idesc1, ks > 0);
                tc::mma_f16kind(tbase + 64, tc::make_desc(opb_u + kTan + tc::kmajor_off(0, 16 * ks, MD::K1), 128,
                                                       (MD::K1 / 8) * 128), bd, idesc1, ks > 0);
              }
              tc::commit(&mbar);
            }
            MIX_WAIT();
            if (!ok) break;
            if (half == 0)
              emb_epi1<E0, E1, E2, 0, true>(tbase + lane_off, tbase + 64 + lane_off, row, opb, opb + kTan, h0, d0, h1,
                                            d1);
            else
              emb_epi1<E0, E1, E2, 1, true>(tbase + lane_off, tbase + 64 + lane_off, row, opb, opb + kTan, h0, d0, h1,
                                            d1);
          }
          tc::fence_proxy_async();
          tc::fence_before_sync();
          __syncthreads();
          if (warp == 0 && tc::elect_one()) {
            tc::fence_after_sync();
#pragma unroll
            for (int ks = 0; ks < MD::K2 / 16; ++ks) {
              const uint64_t bd = tc::make_desc(w2_u + tc::kmajor_off(0, 16 * ks, MD::K2), 128, (MD::K2 / 8) * 128);
              tc::mma_f16kind(tbase, tc::make_desc(opb_u + tc::kmajor_off(0, 16 * ks, MD::K2), 128,
                                                (MD::K2 / 8) * 128), bd, idesc2, ks > 0);
              tc::mma_f16kind(tbase + 128, tc::make_desc(opb_u + kTan + tc::kmajor_off(0, 16 * ks, MD::K2), 128,
                                                      (MD::K2 / 8) * 128), bd, idesc2, ks > 0);
            }
            tc::commit(&mbar);
          }
          MIX_WAIT();
          if (!ok) break;
          if (half == 0)
            emb_epi2<E0, E1, E2, 0, true>(tbase + lane_off, tbase + 128 + lane_off, opb, opb + kTan, h2off, h1, d1);
          else
            emb_epi2<E0, E1, E2, 1, true>(tbase + lane_off, tbase + 128 + lane_off, opb, opb + kTan, h2off, h1, d1);
          tc::fence_proxy_async();
          tc::fence_before_sync();
          __syncthreads();
          if (warp == 0 && tc::elect_one()) {
            tc::fence_after_sync();
            const uint32_t idesc3 = tc::idesc_f16(128, 16 * (smax - smin + 1), 0, 0);
#pragma unroll
            for (int ks = 0; ks < MD::N2 / 16; ++ks) {
              const uint64_t bd =
                  tc::make_desc(dtb_u + tc::kmajor_off(16 * smin, 16 * ks, MD::N2), 128, (MD::N2 / 8) * 128);
              tc::mma_f16kind(tbase, tc::make_desc(opb_u + tc::kmajor_off(0, 16 * ks, MD::N2), 128,
                                                (MD::N2 / 8) * 128), bd, idesc3, ks > 0);
              tc::mma_f16kind(tbase + 128, tc::make_desc(opb_u + kTan + tc::kmajor_off(0, 16 * ks, MD::N2), 128,
                                                      (MD::N2 / 8) * 128), bd, idesc3, ks > 0);
            }
            tc::commit(&mbar);
          }
          MIX_WAIT();
          if (!ok) break;
          // ---- u, v of this row's slot: the warp loads the 16-column block of
          // each slot among its rows (sorted, so one or two blocks)
          const int packed = act ? __float_as_int(rv.w) : 0;
          const int slot = packed & 7, jsrc = packed >> 3;
          const int wmin = __reduce_min_sync(0xffffffffu, act ? slot : 7);
          const int wmax = __reduce_max_sync(0xffffffffu, act ? slot : 0);
          float u[10], v[10];
#pragma unroll
          for (int c = 0; c < 10; ++c) u[c] = v[c] = 0.f;
          for (int uv = 0; uv < 2; ++uv)
            for (int sl = wmin; sl <= wmax; ++sl) {
              uint32_t r16[16];
              tc::tmem_ld16_issue(tbase + 128 * uv + lane_off + (uint32_t)(16 * (sl - smin)), r16);
              tc::tmem_wait();
              if (slot == sl) {
#pragma unroll
                for (int c = 0; c < 10; ++c) {
                  if (uv == 0) u[c] = __uint_as_float(r16[c]);
                  else v[c] = __uint_as_float(r16[c]);
                }
              }
            }
          tc::fence_before_sync();
          RowGeom gm;
          float gst = 0.f;
          {
            float st2, R[10];
            mix_row_env(rv, M.rcut, inv_std, mean, gm, st2, R);
#pragma unroll
            for (int c = 0; c < 10; ++c) gst = fmaf(R[c], v[c], gst);
          }
          float gx[3];
          row_adjoint_mixed(gm, inv_std, u, gst, gx);
          const float scl = act ? sc_s[slot] : 0.f;  // undo the atom's dE/dT scale
          gx[0] *= scl;
          gx[1] *= scl;
          gx[2] *= scl;
          if (half == 0) {
            if (act) {
              force_add(F4[frame_base + jsrc], -gx[0], -gx[1], -gx[2]);
#pragma unroll
              for (int p3 = 0; p3 < 3; ++p3)
#pragma unroll
                for (int q3 = 0; q3 < 3; ++q3) vir[p3 * 3 + q3] -= gm.x[p3] * gx[q3];
            }
          } else {
            // centre-atom force: the warp's rows are sorted by slot, so a
            // segmented suffix sum leaves each slot's total on its first lane
            const int key = act ? slot : -1 - lane;
            float s0 = gx[0], s1 = gx[1], s2 = gx[2];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
              const int ko = __shfl_down_sync(0xffffffffu, key, o);
              const float t0 = __shfl_down_sync(0xffffffffu, s0, o);
              const float t1 = __shfl_down_sync(0xffffffffu, s1, o);
              const float t2 = __shfl_down_sync(0xffffffffu, s2, o);
              if (lane + o < 32 && ko == key) { s0 += t0; s1 += t1; s2 += t2; }
            }
            const int kp = __shfl_up_sync(0xffffffffu, key, 1);
            if (act && (lane == 0 || kp != key)) {
              force_add(F4[frame_base + src_s[slot]], s0, s1, s2);
            }
          }
          rowstart += nrows;
        }
      }
    }
    if (!ok) break;
    tc::cp_async_wait<0>();
    __syncthreads();
  }
#pragma unroll
  for (int k = 0; k < 9; ++k) {
    const float s = warp_sum(vir[k]);
    if (lane == 0 && s != 0.f) atomicAdd(&vir_s[k], (double)s);
  }
  if (!ok) {
    if (tid == 0) atomicOr(err, 1);
    tc::mbar_wait(&mbar, ph);
  }
  tc::cp_async_wait<0>();
  tc::fence_before_sync();
  __syncthreads();
  if (tid < 9 && vframe >= 0) atomicAdd(&virial[vframe * 9 + tid], vir_s[tid]);
  if (warp == 0) tc::tmem_dealloc(tbase, 256);
}

template <int E0, int E1, int E2>
size_t mix_bwd_smem() {
  using MD = MixDims<E0, E1, E2>;
  return (size_t)round1k(MD::NETB) + round1k(MD::NSMALL * 4) + round1k(kDtbRows * MD::N2 * 2) +
         round1k(2 * MD::OPA) + kRowCapBwd * 16;
}

template <int E0, int E1, int E2>
int launch_mix_embed_bwd(const DevModel &M, const SysDesc &D, const float4 *posS,
                         const float *box, const int32_t *nbrs, const __half *dTh, const float *dTs,
                         const float4 *rows_g, const int *rcnt, ForceSum *F4, double *virial, int *err,
                         cudaStream_t st) {
  // one launch over every centre type and frame: a CTA's blocks run through the
  // frames of a type in increasing order, and it flushes its virial sum to a
  // frame's row before it moves on to the next frame (flush_virial)
  const int nblk = blocks_total(D, kBlkAtoms);
  if (nblk == 0) return DPB_OK;
  const size_t smem = mix_bwd_smem<E0, E1, E2>();
  DPB_CUDA_TRY(cudaFuncSetAttribute(k_mix_embed_bwd<E0, E1, E2>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)smem));
  const int grid = nblk < 2 * num_sms() ? nblk : 2 * num_sms();
  k_mix_embed_bwd<E0, E1, E2><<<grid, kBwdThreads, smem, st>>>(M, D, posS, box, nbrs, dTh, dTs, rows_g, rcnt, F4,
                                                                virial, err);
  count_launch();
  DPB_LAUNCH_CHECK();
  return DPB_OK;
}

// ---------------------------------------------------------------- fitting chain (FP16 tcgen05, TMA weights)
// One CTA per 128 atoms of one centre type (thread = atom = TMEM lane).  The
// forward layers, the adjoint down to the first hidden layer and dE/dG are a
// fixed sequence of M = 128 GEMMs on the tensor cores, with L hidden layers:
//   g <  L           forward layer g        A: G rows (g = 0) or H    B: W_g^T  (out x in)
//   L <= g < 2L - 1  adjoint layer 2L-1-g   A: gZ                     B: W_l    (in x out)
//   g >= 2L - 1      dE/dG columns [128 p, 128 p + 128), p = g - (2L - 1), B: rows of W_0
// Warp roles (320 threads): warps 0-7 are the epilogue, two threads per atom
// (warps w and w + 4 share TMEM lane quarter w and take the two halves of
// every layer's columns), which also stream layer 0's G rows; one
// thread of warp 8 issues the MMAs and one of warp 9 the bulk (TMA) copies of
// the weights, each waiting only on its own barriers so MMAs queue back to
// back.  The weights pass through a ring of stages of KC K = 16 steps (full /
// empty mbarriers), so those of the next GEMM are already in flight while the
// epilogue of the current one runs; layer 0's A operand passes through a second
// ring in the space that the activations take later.  The dE/dG passes
// alternate between two TMEM accumulators so that the epilogue of pass p
// overlaps the MMAs of pass p + 1.
// A K = 16 step of the weights is [k8 (2)][row][8 fp16] (K-major core matrices,
// no swizzle: LBO = rows x 16 B between the two K halves, SBO = 128 B between
// 8-row groups).  The weights are stored pre-tiled in exactly this
// layout (DevModel::fit_bt, built at model creation), so a stage is one
// contiguous cp.async.bulk.
// Epilogues run in FP32 on the CUDA cores: tanh, dt-residuals, the energy dot
// product (FP64 segment sums) and the adjoint gates; tanh values and residual
// sources go to a per-atom FP32 scratch, the FP16 activation of the next GEMM
// stays in shared memory, as do the biases, dt and output weights.
//
// What bounds it: the chain of a tile, GEMM after epilogue.  One tile of width 240
// and K0 = 1600 took 153 us: the single issuing thread spent 470 clocks per step
// on its wait and MMA (branches and uniform operands serialised, see
// tc::elect_one), layer 0's ring ran empty at every stage, and each 8 columns of
// an epilogue waited on L2 for 32 bytes of biases.  It takes 80 us: layer 0 16,
// the six hidden GEMMs and epilogues 6 each, the dE/dG passes 25.  98,304 atoms
// took 609 us and take 505 us.
constexpr int kFitThreads = 320;
constexpr int kFitEpi = 256;                 // epilogue threads: 2 per atom
constexpr int kFitDgN = 128;                 // N of one dE/dG pass
constexpr int kFitStepA = 2 * 128 * 16;      // A bytes of a K = 16 step

// Pipeline shape: the shallow one (stages of two steps) fits two CTAs per SM
// (one CTA's epilogue overlaps the other's MMAs); the deep one has stages of
// four steps and more weights in flight, for one CTA per SM.  dpb_md_autotune
// times both.
template <int FW, bool DEEP>
struct FitCfg {
  static constexpr int BR = FW > kFitDgN ? FW : kFitDgN;  // rows of the largest B box
  static constexpr int KC = DEEP ? 4 : 2;                 // K = 16 steps per stage
  static constexpr int STAGE = KC * BR * 32, STAGEA = KC * kFitStepA;
  static constexpr int HAB = 128 * FW * 2;
  static constexpr int RA = HAB > 3 * STAGEA ? HAB : 3 * STAGEA;  // activations, and layer 0's A ring
  static constexpr int NA = RA / STAGEA < 8 ? RA / STAGEA : 8;
  static constexpr int ST = DEEP ? (FW > 240 ? 4 : 5) : (FW > 240 ? 2 : 3);
  // time of two tiles that share an SM over that of one that has it to itself, in
  // eighths: 1.53 to 1.78 measured for widths 64 and 128 (K0 400 to 1600, one to three
  // layers), 1.72 to 1.93 for 208 to 256 (one to four)
  static constexpr int PAIR8 = FW <= 128 ? 13 : 15;
  // biases of the L layers, dt of layers 1 .. L - 1 (of layer 0 for L = 1), output
  // weights, and the energies that one half of the epilogue hands to the other:
  // these in the biases of layer 0, which are done with then, where they fit
  static __host__ __device__ constexpr int dt_at(int L, int l) { return (L + (L > 1 ? l - 1 : l)) * FW; }
  static __host__ __device__ constexpr int wout_at(int L) { return (L + (L > 1 ? L - 1 : 1)) * FW; }
  static __host__ __device__ constexpr int esum_at(int L) { return L > 1 && FW >= 128 ? 0 : wout_at(L) + FW; }
  static __host__ __device__ constexpr size_t smem(int L) {
    return (size_t)RA + (size_t)ST * STAGE + (size_t)(wout_at(L) + FW + (esum_at(L) ? 128 : 0)) * 4;
  }
  static constexpr int STATIC = 256;  // barriers, TMEM address, flag
  static_assert((2 * ST + 2 * NA + 6) * 8 + 8 <= STATIC, "static shared memory");
  // 1 KB of every CTA is the system's
  static_assert((DEEP ? 1 : 2) * (smem(kMaxFitLayers) + STATIC + 1024) <= 228 * 1024, "CTAs per SM at every depth");
  static_assert(smem(kMaxFitLayers) + STATIC <= 227 * 1024, "fitting ring");
};

// Bounded mbarrier wait that also gives up once another role of the CTA gave
// up (*abort), so every role leaves its loop and reaches the final barrier.
__device__ __forceinline__ bool fit_wait(uint64_t *bar, uint32_t parity, volatile int *abort) {
  const uint32_t a = tc::smem_u32(bar);
  for (int it = 0; it < tc::kWaitLimit; ++it) {
    if (tc::mbar_test(a, parity)) return true;
    if ((it & 31) == 31 && *abort) return false;
  }
  *abort = 1;
  return false;
}

// The same for a whole warp, one lane polling.
__device__ __forceinline__ bool fit_wait_warp(uint64_t *bar, uint32_t parity, volatile int *abort) {
  bool ok = true;
  if ((threadIdx.x & 31) == 0) ok = fit_wait(bar, parity, abort);
  return __all_sync(0xffffffffu, ok);
}

// One arrival per warp, after its lanes' work.  (Polling and arriving by one lane
// instead of all: 49,152 atoms in two CTAs per SM 315 -> 276 us.)
__device__ __forceinline__ void fit_arrive_warp(uint64_t *bar) {
  __syncwarp();
  if ((threadIdx.x & 31) == 0) tc::mbar_arrive(bar);
}

// Epilogue -> issuer hand-over: TMEM reads done, shared-memory operand written.
__device__ __forceinline__ void fit_signal(uint64_t *bar) {
  tc::fence_before_sync();
  tc::fence_proxy_async();
  fit_arrive_warp(bar);
}

struct FitGemm {
  const char *src;  // pre-tiled B chunks of this GEMM, br x 32 bytes each
  int N, nk, br, col;  // MMA N, K chunks, B rows per chunk, TMEM column
};

template <int FW>
__device__ __forceinline__ FitGemm fit_gemm_info(const DevModel &M, int ti, int g, int L, int K0) {
  FitGemm G;
  if (g < L) {
    G.src = reinterpret_cast<const char *>(M.fit_bt[ti][kFitBtFwd + g]);
    G.N = FW; G.nk = (g == 0 ? K0 : FW) / 16; G.br = FW; G.col = 0;
  } else if (g < 2 * L - 1) {
    G.src = reinterpret_cast<const char *>(M.fit_bt[ti][kFitBtAdj + 2 * L - 1 - g]);
    G.N = FW; G.nk = FW / 16; G.br = FW; G.col = 0;
  } else {
    const int p = g - (2 * L - 1);
    G.nk = FW / 16; G.br = kFitDgN;
    G.src = reinterpret_cast<const char *>(M.fit_bt[ti][kFitBtDg]) + (size_t)p * G.nk * kFitDgN * 32;
    G.N = min(kFitDgN, K0 - kFitDgN * p);
    G.col = kFitDgN * (p & 1);
  }
  return G;
}

// The 128-row tiles of every centre type in one launch: t0[k] is the first tile
// of the k-th type present, ti[k] its index.
struct FitTiles {
  int n, ti[kMaxTypes], t0[kMaxTypes + 1], rows[kMaxTypes];
  RowMap rm[kMaxTypes];
};

template <int FW, typename DGT, bool DEEP>
__global__ void __launch_bounds__(kFitThreads, DEEP ? 1 : 2) k_mix_fit(DevModel M, FitTiles ft,
                                                           const __half *__restrict__ Gh,
                                                           DGT *__restrict__ dGout, float *__restrict__ scratch,
                                                           float *__restrict__ Eatom, double *__restrict__ energy,
                                                           int N, int *__restrict__ err,
                                                           const int32_t *__restrict__ seg) {
  using C = FitCfg<FW, DEEP>;
  constexpr int ST = C::ST, KC = C::KC, NA = C::NA;
  static_assert(FW % 16 == 0 && FW <= 256, "fit width");
  // (an alignment of 1 KB here or in another kernel of this file would round every
  // kernel's static part up to it)
  extern __shared__ __align__(128) char smem[];
  char *HA = smem;              // 128 x FW fp16, K-major (kmajor_off); during layer 0 its A ring
  char *ring = smem + C::RA;    // ST stages
  float *cst = reinterpret_cast<float *>(ring + ST * C::STAGE);  // bias[l], dt[l], w_out, energies
  __shared__ __align__(8) uint64_t full[ST], empty[ST], fullA[NA], emptyA[NA], accf, accfD[2], epid, accfree[2];
  __shared__ uint32_t tbase_s;
  __shared__ int abort_s;
  const int tid = threadIdx.x, warp = tc::warp_index();
  const int L = M.nfit, K0 = M.A * M.E2;
  float *esum_s = cst + C::esum_at(L);  // the second half's energy partial per atom
  const int NG = 2 * L - 1 + (K0 + kFitDgN - 1) / kFitDgN;
  volatile int *abort = &abort_s;
  if (tid == 0) {
    for (int s = 0; s < ST; ++s) {
      tc::mbar_init(&full[s], 1);
      tc::mbar_init(&empty[s], 1);
    }
    for (int s = 0; s < NA; ++s) {
      tc::mbar_init(&fullA[s], kFitEpi / 32);
      tc::mbar_init(&emptyA[s], 1);
    }
    tc::mbar_init(&accf, 1);
    tc::mbar_init(&accfD[0], 1);
    tc::mbar_init(&accfD[1], 1);
    tc::mbar_init(&epid, kFitEpi / 32);
    tc::mbar_init(&accfree[0], kFitEpi / 32);
    tc::mbar_init(&accfree[1], kFitEpi / 32);
    abort_s = 0;
    tc::fence_mbar_init();
  }
  int tk = 0;
#pragma unroll
  for (int k = 1; k < kMaxTypes; ++k)
    if (k < ft.n && (int)blockIdx.x >= ft.t0[k]) tk = k;
  const int ti = ft.ti[tk];
  const RowMap rm = ft.rm[tk];
  static_assert(FW <= kFitThreads, "one column per thread");
  if (tid < FW) {  // every load in flight before the first store
    float v[2 * kMaxFitLayers + 1];
#pragma unroll
    for (int l = 0; l < kMaxFitLayers; ++l) {
      v[2 * l] = l < L ? M.mfb[ti][l][tid] : 0.f;
      v[2 * l + 1] = l < L && M.mfdt[ti][l] ? M.mfdt[ti][l][tid] : 1.f;
    }
    v[2 * kMaxFitLayers] = M.mfwout[ti][tid];
#pragma unroll
    for (int l = 0; l < kMaxFitLayers; ++l)
      if (l < L) {
        cst[l * FW + tid] = v[2 * l];
        if (l > 0 || L == 1) cst[C::dt_at(L, l) + tid] = v[2 * l + 1];
      }
    cst[C::wout_at(L) + tid] = v[2 * kMaxFitLayers];
  }
  if (warp == 0) tc::tmem_alloc(&tbase_s, 256);
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t td = tbase_s;
  const int r0 = ((int)blockIdx.x - ft.t0[tk]) * 128, nrows = min(128, ft.rows[tk] - r0);

  if (warp == 9) {
    // ================= weight producer (one thread): bulk copies into free stages
    if (tc::elect_one()) {
      const uint32_t ring_u = tc::smem_u32(ring);
      int p = 0, s = 0;  // stages filled, current stage
      uint32_t ph = 1;   // parity of its previous use
      bool ok = true;
      for (int g = 0; g < NG && ok; ++g) {
        const FitGemm gi = fit_gemm_info<FW>(M, ti, g, L, K0);
        const char *src = gi.src;
        for (int k = 0; k < gi.nk; k += KC, ++p) {
          if (p >= ST && !(ok = fit_wait(&empty[s], ph, abort))) break;
          const uint32_t bytes = (uint32_t)min(KC, gi.nk - k) * gi.br * 32u;
          tc::mbar_arrive_expect_tx(&full[s], bytes);
          tc::bulk_load(ring_u + s * C::STAGE, src, bytes, &full[s]);
          src += bytes;
          if (++s == ST) {
            s = 0;
            ph ^= 1;
          }
        }
      }
      // copies still in flight only after a give-up: the last ST filled stages
      for (int c = p > ST ? p - ST : 0; c < p; ++c) tc::mbar_wait(&full[c % ST], (c / ST) & 1);
    }
  } else if (warp == 8) {
    // ================= MMA issuer (one thread)
    if (tc::elect_one()) {
      const uint32_t ring_u = tc::smem_u32(ring), ha_u = tc::smem_u32(HA);
      int s = 0, sa = 0;
      uint32_t ph = 0, pha = 0, epid_n = 0;
      bool ok = true, any = false;
      for (int g = 0; g < NG && ok; ++g) {
        const FitGemm gi = fit_gemm_info<FW>(M, ti, g, L, K0);
        if (g >= 1 && g <= 2 * L - 1) {  // A operand (and the accumulator) handed back by the epilogue
          ok = fit_wait(&epid, epid_n & 1, abort);
          ++epid_n;
        } else if (g >= 2 * L + 1) {     // dE/dG pass p reuses the accumulator of pass p - 2
          const int pp = g - (2 * L - 1);
          ok = fit_wait(&accfree[pp & 1], ((pp >> 1) - 1) & 1, abort);
        }
        if (!ok) break;
        tc::fence_after_sync();
        const uint32_t idesc = tc::idesc_f16(128, gi.N, 0, 0), d = td + gi.col, bl = (uint32_t)gi.br * 16,
                       bstep = (uint32_t)gi.br * 32;
        // one stage's steps: A at a0 + j astep
        auto steps = [&](int n, uint32_t a0, uint32_t astep, uint32_t albo, uint32_t asbo, bool acc) {
          const uint32_t b0 = ring_u + s * C::STAGE;
          if (n == KC) {
#pragma unroll
            for (int j = 0; j < KC; ++j)
              tc::mma_f16kind(d, tc::make_desc(a0 + j * astep, albo, asbo), tc::make_desc(b0 + j * bstep, bl, 128), idesc,
                              (j > 0 || acc) ? 1u : 0u);
          } else {
            for (int j = 0; j < n; ++j)
              tc::mma_f16kind(d, tc::make_desc(a0 + j * astep, albo, asbo), tc::make_desc(b0 + j * bstep, bl, 128), idesc,
                              (j > 0 || acc) ? 1u : 0u);
          }
          tc::commit(&empty[s]);
        };
        for (int k = 0; k < gi.nk; k += KC) {
          ok = fit_wait(&full[s], ph, abort) && (g != 0 || fit_wait(&fullA[sa], pha, abort));
          if (!ok) break;
          tc::fence_after_sync();
          any = true;
          const int n = min(KC, gi.nk - k);
          if (g == 0) {
            steps(n, ha_u + sa * C::STAGEA, tc::kmajor_off(0, 16, 16 * KC), 128, 16 * KC * 16, k > 0);
            tc::commit(&emptyA[sa]);
            if (++sa == NA) {
              sa = 0;
              pha ^= 1;
            }
          } else {
            steps(n, ha_u + tc::kmajor_off(0, 16 * k, FW), tc::kmajor_off(0, 16, FW), 128, (FW / 8) * 128, k > 0);
          }
          if (++s == ST) {
            s = 0;
            ph ^= 1;
          }
        }
        if (!ok) break;
        tc::commit(g < 2 * L - 1 ? &accf : &accfD[(g - (2 * L - 1)) & 1]);
      }
      // the last MMAs complete before the CTA exits: the stage before s
      if (any) tc::mbar_wait(&empty[s ? s - 1 : ST - 1], s ? ph : ph ^ 1);
    }
  } else {
    // ================= epilogue warps: two threads per atom = TMEM lane; half
    // h = warp / 4 takes columns [h FH, h FH + FH) of every hidden layer and
    // [64 h, 64 h + 64) of every dE/dG pass
    constexpr int FH = FW / 2;
    static_assert(FH % 8 == 0, "half-width column chunks");
    const int row = tid & 127, half = tid >> 7;
    const bool act = row < nrows;
    const size_t me = rm.atom(act ? r0 + row : r0);
    const uint32_t lane_off = (uint32_t)((warp & 3) * 32) << 16;
    const int cb = half * FH, ce = cb + FH;  // this half's hidden columns
    bool ok = true;
    // ---- layer 0's A operand: an instruction loads 64 bytes of 8 rows (whole
    // sectors, and stores without bank conflicts; a thread per row took 1,700
    // clocks per stage), PF stages ahead in registers.  (With asynchronous copies signalled NA - 1 stages later the
    // ring ran empty at every stage: 2,100 clocks each against 470 of its MMAs.)
    {
      constexpr int PF = 8 / KC;
      const int nk0 = K0 / 16, nst = (nk0 + KC - 1) / KC;
      // instruction q: rows 8 (q & 1) + lane % 8 of the warp's 16, 8-wide K groups 4 (q >> 1) + lane / 8
      const int lane = tid & 31, k8 = lane >> 3, r_first = 16 * warp + (lane & 7);
      const char *grow[2];
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const int r = r_first + 8 * q;
        grow[q] = r < nrows ? reinterpret_cast<const char *>(Gh + rm.atom(r0 + r) * (size_t)K0) + k8 * 16 : nullptr;
      }
      char *dst0 = HA + tc::kmajor_off(r_first, 8 * k8, 16 * KC);
      uint4 v[PF][KC];
      auto load = [&](int c, uint4 (&x)[KC]) {
#pragma unroll
        for (int q = 0; q < KC; ++q)
          x[q] = grow[q & 1] && c * KC + 2 * (q >> 1) + (k8 >> 1) < nk0
                     ? *reinterpret_cast<const uint4 *>(grow[q & 1] + c * KC * 32 + (q >> 1) * 64)
                     : make_uint4(0, 0, 0, 0);
      };
#pragma unroll
      for (int p = 0; p < PF; ++p) load(p, v[p]);
      int s = 0;
      uint32_t ph = 1;  // parity of the stage's previous use
      for (int c0 = 0; c0 < nst && ok; c0 += PF) {
#pragma unroll
        for (int p = 0; p < PF; ++p) {
          const int c = c0 + p;
          if (c >= nst || !ok) continue;
          if (c >= NA && !(ok = fit_wait_warp(&emptyA[s], ph, abort))) continue;
          char *dst = dst0 + s * C::STAGEA;
#pragma unroll
          for (int q = 0; q < KC; ++q)
            *reinterpret_cast<uint4 *>(dst + tc::kmajor_off(8 * (q & 1), 32 * (q >> 1), 16 * KC)) = v[p][q];
          load(c + PF, v[p]);
          tc::fence_proxy_async();
          fit_arrive_warp(&fullA[s]);
          if (++s == NA) {
            s = 0;
            ph ^= 1;
          }
        }
      }
    }
    uint32_t accf_n = 0;
    // per-CTA scratch tile [slot][n][thread] (coalesced): slots 0..L-2 tanh
    // values, L..2L-2 layer outputs (hidden layers below the last), 2L the
    // residual adjoint
    float *tile = scratch + (size_t)blockIdx.x * 128 * (size_t)(2 * L + 1) * FW + row;
#define FIT_SCR(slot, n) tile[((size_t)(slot) * FW + (n)) * 128]
    // L2 prefetch of one scratch slot of this warp's 32 rows and this half's
    // columns (one 128-byte line per column), issued before a layer's
    // accumulator wait so that it overlaps the layer's MMAs
    const float *tile_w = tile - (row & 31);
    auto prefetch_slot = [&](int slot) {
      for (int n = cb + (row & 31); n < ce; n += 32) tc::prefetch_l2(tile_w + ((size_t)slot * FW + n) * 128);
    };
    // ---- forward; the last layer's epilogue also forms the atom energy and
    // the first adjoint gate g = w_out dt (1 - t^2), the A operand of adjoint
    // layer L-1 (its t and h never go to the scratch)
    float e_sum = 0.f;
    for (int l = 0; l < L && ok; ++l) {
      if (M.mfdt[ti][l]) prefetch_slot(M.mfdt[ti][l - 1] ? L + l - 1 : l - 1);
      ok = fit_wait_warp(&accf, accf_n & 1, abort);
      ++accf_n;
      if (!ok) break;
      tc::fence_after_sync();
      const bool last = l == L - 1;
      const float *dt = M.mfdt[ti][l];
      const float usc = 1.f / M.fit_wsc[ti][l];         // a power of two: exact
      const float gsc = last ? M.fit_gsc[ti][l] : 1.f;  // the gate's operand scale
      // residual sources of two chunks of 8 columns, each reloaded for the chunk
      // after next as soon as it is used
      const bool res = dt != nullptr;
      const int hs = res && !M.mfdt[ti][l - 1] ? l - 1 : L + l - 1;  // the layer below's output
      // (layer 0 of several has no dt: it reads there what it does not use)
      const float *cb_ = cst + l * FW, *cd_ = cst + C::dt_at(L, l), *cw_ = cst + C::wout_at(L);
      float hp[2][8];
#pragma unroll
      for (int q = 0; q < 2; ++q)
#pragma unroll
        for (int i = 0; i < 8; ++i) hp[q][i] = (res && cb + 8 * q < ce) ? FIT_SCR(hs, cb + 8 * q + i) : 0.f;
      auto chunk = [&](int c0, const uint32_t (&r)[8], float (&h_prev)[8]) {
        float hv[8];
#pragma unroll
        for (int q = 0; q < 8; q += 4) {
          const float4 b4 = *reinterpret_cast<const float4 *>(cb_ + c0 + q);
          const float4 d4 = *reinterpret_cast<const float4 *>(cd_ + c0 + q);
          const float4 w4 = last ? *reinterpret_cast<const float4 *>(cw_ + c0 + q) : make_float4(0.f, 0.f, 0.f, 0.f);
          const float bv[4] = {b4.x, b4.y, b4.z, b4.w}, dv[4] = {d4.x, d4.y, d4.z, d4.w},
                      wv[4] = {w4.x, w4.y, w4.z, w4.w};
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int i = q + e, n = c0 + i;
            const float t = tc::tanh_fast(fmaf(__uint_as_float(r[i]), usc, bv[e]));
            float h = t;
            if (res) h = t * dv[e] + h_prev[i];
            if (!last) {
              hv[i] = h;
              FIT_SCR(l, n) = t;
              if (res) FIT_SCR(L + l, n) = h;  // without a residual h is t
            } else {
              e_sum = fmaf(h, wv[e], e_sum);
              hv[i] = wv[e] * dv[e] * (1.f - t * t);
            }
          }
        }
        if (res && c0 + 16 < ce) {
#pragma unroll
          for (int i = 0; i < 8; ++i) h_prev[i] = FIT_SCR(hs, c0 + 16 + i);
        }
        *reinterpret_cast<uint4 *>(HA + tc::kmajor_off(row, c0, FW)) = pack8h(hv, gsc);
      };
      for (int c0 = cb; c0 < ce; c0 += 16) {
        uint32_t ra[8], rb[8];
        tc::tmem_ld8_issue(td + lane_off + c0, ra);
        if (c0 + 8 < ce) tc::tmem_ld8_issue(td + lane_off + c0 + 8, rb);
        tc::tmem_wait();
        chunk(c0, ra, hp[0]);
        if (c0 + 8 < ce) chunk(c0 + 8, rb, hp[1]);
      }
      fit_signal(&epid);
    }
    // the two halves' energy partials (every epilogue thread reaches this
    // barrier once, whatever its wait outcomes)
    if (half) esum_s[row] = e_sum;
    asm volatile("bar.sync 1, %0;" ::"n"(kFitEpi) : "memory");
    if (half == 0) {
      float e_me = 0.f;
      if (ok) {
        e_me = e_sum + esum_s[row] + M.fb[ti][L][0];
        if (act) Eatom[me] = e_me;
      }
      // energy per segment (every lane of the warp takes part): rows run
      // through the segments in order, so a warp suffix sum over equal keys
      // leaves each run's total at its first lane
      const int lane = row & 31;
      const int key = (ok && act) ? energy_slot(seg, me, N) : -2;
      double v = (ok && act) ? (double)e_me : 0.0;
#pragma unroll
      for (int off = 1; off < 32; off <<= 1) {
        const double o = __shfl_down_sync(0xffffffffu, v, off);
        const int ko = __shfl_down_sync(0xffffffffu, key, off);
        if (lane + off < 32 && ko == key) v += o;
      }
      const int kprev = __shfl_up_sync(0xffffffffu, key, 1);
      if (key >= 0 && (lane == 0 || kprev != key)) atomicAdd(&energy[key], v);
    }
    // ---- adjoint: layers L-1 .. 1, gH_{l-1} = gZ_l W_l^T (+ gH_l if residual)
    for (int l = L - 1; l >= 1 && ok; --l) {
      if (M.mfdt[ti][l] != nullptr && l != L - 1) prefetch_slot(2 * L);
      prefetch_slot(l - 1);
      ok = fit_wait_warp(&accf, accf_n & 1, abort);
      ++accf_n;
      if (!ok) break;
      tc::fence_after_sync();
      const bool res_l = M.mfdt[ti][l] != nullptr, res_lm1 = (l - 1 > 0) && M.mfdt[ti][l - 1] != nullptr;
      const bool use_gh = res_l && l != L - 1;
      const float usc = 1.f / (M.fit_wsc[ti][l] * M.fit_gsc[ti][l]), gsc = M.fit_gsc[ti][l - 1];
      // dt of layer l - 1 (1 without residual), output weights
      const float *cd_ = cst + C::dt_at(L, l - 1), *cw_ = cst + C::wout_at(L);
      float ghc[2][8], tcur[2][8];
#pragma unroll
      for (int q = 0; q < 2; ++q)
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const bool in = cb + 8 * q < ce;
          ghc[q][i] = (use_gh && in) ? FIT_SCR(2 * L, cb + 8 * q + i) : 0.f;
          tcur[q][i] = in ? FIT_SCR(l - 1, cb + 8 * q + i) : 0.f;
        }
      auto chunk = [&](int c0, const uint32_t (&r)[8], float (&gh)[8], float (&tt)[8]) {
        float gz[8];
#pragma unroll
        for (int q = 0; q < 8; q += 4) {
          const float4 w4 = *reinterpret_cast<const float4 *>(cw_ + c0 + q);
          const float4 d4 = res_lm1 ? *reinterpret_cast<const float4 *>(cd_ + c0 + q) : make_float4(1.f, 1.f, 1.f, 1.f);
          const float wv[4] = {w4.x, w4.y, w4.z, w4.w}, dv[4] = {d4.x, d4.y, d4.z, d4.w};
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int i = q + e, n = c0 + i;
            float g = __uint_as_float(r[i]) * usc;
            if (res_l) g += (l == L - 1) ? wv[e] : gh[i];
            const float t = tt[i];
            gz[i] = g * dv[e] * (1.f - t * t);
            if (res_lm1) FIT_SCR(2 * L, n) = g;
          }
        }
        if (c0 + 16 < ce) {
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            if (use_gh) gh[i] = FIT_SCR(2 * L, c0 + 16 + i);
            tt[i] = FIT_SCR(l - 1, c0 + 16 + i);
          }
        }
        *reinterpret_cast<uint4 *>(HA + tc::kmajor_off(row, c0, FW)) = pack8h(gz, gsc);
      };
      for (int c0 = cb; c0 < ce; c0 += 16) {
        uint32_t ra[8], rb[8];
        tc::tmem_ld8_issue(td + lane_off + c0, ra);
        if (c0 + 8 < ce) tc::tmem_ld8_issue(td + lane_off + c0 + 8, rb);
        tc::tmem_wait();
        chunk(c0, ra, ghc[0], tcur[0]);
        if (c0 + 8 < ce) chunk(c0 + 8, rb, ghc[1], tcur[1]);
      }
      fit_signal(&epid);
    }
    // ---- dE/dG = gZ_0 W_0^T, 128 columns per pass from alternating
    // accumulators, this half's 64 of them
    const int npass = (K0 + kFitDgN - 1) / kFitDgN;
    const float usc0 = 1.f / (M.fit_wsc[ti][0] * M.fit_gsc[ti][0]);
    for (int pp = 0; pp < npass && ok; ++pp) {
      ok = fit_wait_warp(&accfD[pp & 1], (pp >> 1) & 1, abort);
      if (!ok) break;
      tc::fence_after_sync();
      const int n0 = kFitDgN * pp, nv = min(kFitDgN, K0 - n0);
      const uint32_t tcol = td + lane_off + kFitDgN * (pp & 1);
      for (int c0 = 64 * half; c0 < min(nv, 64 * half + 64); c0 += 32) {
        const bool two = c0 + 16 < nv;
        uint32_t ra[16], rb[16];
        tc::tmem_ld16_issue(tcol + c0, ra);
        if (two) tc::tmem_ld16_issue(tcol + c0 + 16, rb);
        tc::tmem_wait();
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          ra[i] = __float_as_uint(__uint_as_float(ra[i]) * usc0);
          rb[i] = __float_as_uint(__uint_as_float(rb[i]) * usc0);
        }
        if (act) {
          if constexpr (sizeof(DGT) == 4) {  // FP32 (for the FP32 embedding adjoint)
            float4 *dst = reinterpret_cast<float4 *>(dGout + me * K0 + n0 + c0);
#pragma unroll
            for (int i = 0; i < 16; i += 4)
              dst[i / 4] = make_float4(__uint_as_float(ra[i]), __uint_as_float(ra[i + 1]),
                                       __uint_as_float(ra[i + 2]), __uint_as_float(ra[i + 3]));
            if (two) {
#pragma unroll
              for (int i = 0; i < 16; i += 4)
                dst[4 + i / 4] = make_float4(__uint_as_float(rb[i]), __uint_as_float(rb[i + 1]),
                                             __uint_as_float(rb[i + 2]), __uint_as_float(rb[i + 3]));
            }
          } else {  // FP16 times fit_dgsc (for the tensor-core embedding adjoint)
            float fa[16], fb[16];
#pragma unroll
            for (int i = 0; i < 16; ++i) {
              fa[i] = __uint_as_float(ra[i]);
              fb[i] = __uint_as_float(rb[i]);
            }
            const float dgsc = M.fit_dgsc;
            uint4 *dst = reinterpret_cast<uint4 *>(dGout + me * K0 + n0 + c0);
            dst[0] = pack8h(fa, dgsc);
            dst[1] = pack8h(fa + 8, dgsc);
            if (two) {
              dst[2] = pack8h(fb, dgsc);
              dst[3] = pack8h(fb + 8, dgsc);
            }
          }
        }
      }
      tc::fence_before_sync();
      fit_arrive_warp(&accfree[pp & 1]);
    }
#undef FIT_SCR
  }
  tc::cp_async_wait<0>();
  tc::fence_before_sync();
  __syncthreads();
  if (tid == 0 && abort_s) atomicOr(err, 1);
  if (warp == 0) tc::tmem_dealloc(td, 256);
}

template <int FW, typename DGT, bool DEEP>
int launch_mix_fit(const DevModel &M, const SysDesc &D, const __half *Gb, DGT *dG, float *scratch,
                   float *Eatom, double *energy, int *err, cudaStream_t st) {
  using C = FitCfg<FW, DEEP>;
  if (!M.fit_bt[0][kFitBtDg]) return DPB_ERR_UNSUPPORTED;
  DPB_CUDA_TRY(
      cudaFuncSetAttribute(k_mix_fit<FW, DGT, DEEP>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::smem(M.nfit)));
  FitTiles ft{};  // scratch tiles of 128 rows are numbered as the launch's tiles
  for (int ti = 0; ti < M.ntypes; ++ti) {
    const int cnt = D.offs[ti + 1] - D.offs[ti];
    if (!cnt) continue;
    ft.ti[ft.n] = ti;
    ft.rm[ft.n] = RowMap{cnt, D.N, D.offs[ti]};
    ft.rows[ft.n] = cnt * D.F;
    ft.t0[ft.n + 1] = ft.t0[ft.n] + (cnt * D.F + 127) / 128;
    ++ft.n;
  }
  if (ft.n == 0) return DPB_OK;
  k_mix_fit<FW, DGT, DEEP><<<ft.t0[ft.n], kFitThreads, C::smem(M.nfit), st>>>(M, ft, Gb, dG, scratch, Eatom, energy, D.N, err,
                                                                      D.seg);
  count_launch();
  DPB_LAUNCH_CHECK();
  return DPB_OK;
}

// The instantiation of the model's padded hidden width and ring depth.
template <int FW, typename DGT>
static int launch_mix_fit_d(const DevModel &M, const SysDesc &D, const __half *Gb, DGT *dG, float *scratch,
                            float *Eatom, double *energy, int *err, FitShape shape, cudaStream_t st) {
  // unless timed for this many tiles, the shape whose whole waves take less
  int cnt[kMaxTypes];
  for (int ti = 0; ti < M.ntypes; ++ti) cnt[ti] = D.offs[ti + 1] - D.offs[ti];
  const int tiles = fit_tiles(M.ntypes, cnt, D.F), sms = num_sms();
  const bool deep = shape.deep >= 0 && shape.tiles == tiles
                        ? shape.deep != 0
                        : 8 * ((tiles + sms - 1) / sms) <
                              FitCfg<FW, false>::PAIR8 * ((tiles + 2 * sms - 1) / (2 * sms));
  return deep ? launch_mix_fit<FW, DGT, true>(M, D, Gb, dG, scratch, Eatom, energy, err, st)
              : launch_mix_fit<FW, DGT, false>(M, D, Gb, dG, scratch, Eatom, energy, err, st);
}

template <typename DGT>
int launch_mix_fit_any(const DevModel &M, const SysDesc &D, const __half *Gb, DGT *dG, float *scratch,
                       float *Eatom, double *energy, int *err, FitShape shape, cudaStream_t st) {
  switch (M.mfw) {
    case 64: return launch_mix_fit_d<64, DGT>(M, D, Gb, dG, scratch, Eatom, energy, err, shape, st);
    case 128: return launch_mix_fit_d<128, DGT>(M, D, Gb, dG, scratch, Eatom, energy, err, shape, st);
    case 208: return launch_mix_fit_d<208, DGT>(M, D, Gb, dG, scratch, Eatom, energy, err, shape, st);
    case 240: return launch_mix_fit_d<240, DGT>(M, D, Gb, dG, scratch, Eatom, energy, err, shape, st);
    case 256: return launch_mix_fit_d<256, DGT>(M, D, Gb, dG, scratch, Eatom, energy, err, shape, st);
    default: return DPB_ERR_UNSUPPORTED;
  }
}

// ---------------------------------------------------------------- dispatch
// Hidden widths with a tensor-core fitting instantiation; a model's hidden
// layers all run at the smallest one that holds its widest layer.
static const int kFitWidths[] = {64, 128, 208, 240, 256};

int mixed_fit_width(const DevModel &M) {
  int w = 0;
  for (int l = 0; l < M.nfit; ++l) w = w > M.FW[l] ? w : M.FW[l];
  for (int c : kFitWidths)
    if (w <= c) return c;
  return 0;
}

// The mixed form needs the tensor-core fitting (padded width, dE/dG passes of
// whole 16-column chunks); the embedding runs on the tensor cores for the
// tuned shapes and in the FP32 kernels otherwise.
int mixed_supported(const DevModel &M) { return M.mfw > 0 && (M.A * M.E2) % 16 == 0; }

static size_t al256(size_t x) { return (x + 255) & ~(size_t)255; }

static int n2_of(const DevModel &M) { return (M.E2 + 15) / 16 * 16; }

// Fitting scratch rounds each centre type's rows up to whole 128-row tiles.
size_t mixed_workspace_fixed(const DevModel &M) {
  return (size_t)127 * M.ntypes * (2 * M.nfit + 1) * M.mfw * 4 + 1024;
}

size_t mixed_workspace_per_atom(const DevModel &M) {
  const int FW = M.mfw, K0 = M.A * M.E2;
  return (size_t)10 * M.E2 * 4 + (size_t)K0 * 2 + (size_t)K0 * 4 + (size_t)10 * n2_of(M) * 2 + 4 + 16 +
         (size_t)kRowStoreCap * 16 + (size_t)M.ntypes * 4 + (size_t)(2 * M.nfit + 1) * FW * 4 + 48;
}

// dE/dT with W atoms (warps) per block, W in {2, 4, 8} (launch shape only).
template <int E2, int N2, int W>
static void launch_mix_dT_s(const DevModel &M, size_t NF, const float *T, const __half *dGb, __half *dTh,
                            float *dTs, cudaStream_t st) {
  // warp-strided atoms, as many blocks as the SMs hold: a warp zeroes its tiles once
  // and loads one atom ahead (more blocks than are resident, so two or three atoms
  // per warp: 280 us for 98,304 atoms at W = 4, 261 us now)
  constexpr int smem = W * DtCfg<E2, N2>::WARP_BYTES;
  static const int per_sm = [] {  // registers are given to warps in units of 256, on four schedulers of 16,384
    cudaFuncAttributes fa;
    if (cudaFuncGetAttributes(&fa, k_mix_dT<E2, N2, W>) != cudaSuccess) return 1;
    const int warps = 4 * (16384 / ((fa.numRegs + 7) / 8 * 256));
    return std::max(1, std::min({warps / W, 64 / W, 228 * 1024 / (smem + 1024)}));
  }();
  const unsigned grid = (unsigned)std::min((NF + W - 1) / W, (size_t)num_sms() * per_sm);
  cudaFuncSetAttribute(k_mix_dT<E2, N2, W>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  k_mix_dT<E2, N2, W><<<grid, 32 * W, smem, st>>>(M, (int)NF, T, dGb, dTh, dTs);
  count_launch();
}

template <int W>
static void launch_mix_dT_w(const DevModel &M, size_t NF, const float *T, const __half *dGb,
                            __half *dTh, float *dTs, cudaStream_t st) {
  if (M.E2 == 100) launch_mix_dT_s<100, 112, W>(M, NF, T, dGb, dTh, dTs, st);
  else launch_mix_dT_s<64, 64, W>(M, NF, T, dGb, dTh, dTs, st);
}

static int launch_mix_dT(const DevModel &M, size_t NF, const float *T, const __half *dGb, __half *dTh,
                         float *dTs,
                         int warps, cudaStream_t st) {
  switch (warps) {
    case 2: launch_mix_dT_w<2>(M, NF, T, dGb, dTh, dTs, st); break;
    case 8: launch_mix_dT_w<8>(M, NF, T, dGb, dTh, dTs, st); break;
    default: launch_mix_dT_w<4>(M, NF, T, dGb, dTh, dTs, st); break;
  }
  DPB_LAUNCH_CHECK();
  return DPB_OK;
}

// rows / rcnt (may be null): the row store, built here by k_rows and
// streamed by the forward and the adjoint embedding kernels.
int mixed_descriptors(const DevModel &M, const SysDesc &D, const float4 *posS, const float *box,
                      const int32_t *nbrs, float *T, __half *Gb, float4 *rows, int *rcnt, int *err,
                      cudaStream_t st) {
  if (M.ngrids > 0 || !M.emb_tuned) return DPB_ERR_UNSUPPORTED;  // the FP32 kernels give T and G
  prof_begin(PROF_MIXED_EMBED_FWD, st);
  if (rows) {
    const int rc = launch_rows(M, D, kBlkAtoms, posS, box, nbrs, rows, rcnt, st);
    if (rc) return rc;
  }
  const int rc = (M.E2 == 100)
                     ? launch_mix_embed_fwd<25, 50, 100>(M, D, posS, box, nbrs, T, Gb, rows, rcnt, err, st)
                     : launch_mix_embed_fwd<32, 32, 64>(M, D, posS, box, nbrs, T, Gb, rows, rcnt, err, st);
  if (rc) return rc;
  prof_end(PROF_MIXED_EMBED_FWD, st);
  return DPB_OK;
}

__global__ void k_f16_to_f32(const __half *__restrict__ a, float *__restrict__ b, size_t n) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) b[i] = __half2float(a[i]);
}

// FP32 -> FP16 rounded to nearest, without saturation (as the embedding
// kernel writes G).
__global__ void k_f32_to_f16(const float4 *__restrict__ a, uint2 *__restrict__ b, size_t n4) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n4) {
    const float4 v = a[i];
    b[i] = make_uint2(tc::as_u32(__floats2half2_rn(v.x, v.y)), tc::as_u32(__floats2half2_rn(v.z, v.w)));
  }
}

template <int E2>
int launch_embed_fwd_cmp(const DevModel &M, const SysDesc &D, int ti, const float *pos, const int32_t *perm,
                         const float *box, const int32_t *nbrs, float *T, float *G, float *gmax, cudaStream_t st);
template <int E2>
int launch_embed_bwd_cmp(const DevModel &M, const SysDesc &D, int ti, const float *pos, const int32_t *perm,
                         const float *box, const int32_t *nbrs, const float *T, const float *dG, ForceSum *F4,
                         double *virial, cudaStream_t st);
int launch_embed_fwd_gen(const DevModel &, const SysDesc &, int, const float *, const int32_t *, const float *,
                         const int32_t *, float *, float *, float *, cudaStream_t);
int launch_embed_bwd_gen(const DevModel &, const SysDesc &, int, const float *, const int32_t *, const float *,
                         const int32_t *, const float *, const float *, ForceSum *, double *, cudaStream_t);

// Embedding nets without tensor-core kernels in the mixed form - compressed
// tables (a lookup, no GEMM) and shapes other than the tuned ones: the FP32
// kernels produce T and G (FP32) and take the adjoint; the fitting chain runs
// on the tensor cores from an FP16 copy of G.
static int mixed_eval_compressed(const DevModel &M, const SysDesc &D, const float *pos, const int32_t *perm,
                                 const float *box, const int32_t *nbrs, double *energy, float *Eatom, ForceSum *F4,
                                 double *virial, float *T, __half *Gb, float *dG, float *scratch, int *err,
                                 FitShape fit, cudaStream_t st) {
  const size_t NF = (size_t)D.N * D.F;
  const size_t NG = NF * M.A * M.E2;  // a multiple of 16 (mixed_supported)
  int rc;
  prof_begin(PROF_EMBED_FWD, st);
  for (int ti = 0; ti < M.ntypes; ++ti) {
    rc = !M.emb_tuned   ? launch_embed_fwd_gen(M, D, ti, pos, perm, box, nbrs, T, dG, nullptr, st)
         : M.E2 == 100 ? launch_embed_fwd_cmp<100>(M, D, ti, pos, perm, box, nbrs, T, dG, nullptr, st)
                       : launch_embed_fwd_cmp<64>(M, D, ti, pos, perm, box, nbrs, T, dG, nullptr, st);
    if (rc) return rc;
  }
  k_f32_to_f16<<<(unsigned)((NG / 4 + 255) / 256), 256, 0, st>>>(reinterpret_cast<const float4 *>(dG),
                                                                   reinterpret_cast<uint2 *>(Gb), NG / 4);
  count_launch();
  DPB_LAUNCH_CHECK();
  prof_end(PROF_EMBED_FWD, st);
  prof_begin(PROF_MIXED_FIT, st);
  rc = launch_mix_fit_any<float>(M, D, Gb, dG, scratch, Eatom, energy, err, fit, st);
  prof_end(PROF_MIXED_FIT, st);
  if (rc) return rc;
  prof_begin(PROF_EMBED_BWD, st);
  for (int ti = 0; ti < M.ntypes; ++ti) {
    rc = !M.emb_tuned   ? launch_embed_bwd_gen(M, D, ti, pos, perm, box, nbrs, T, dG, F4, virial, st)
         : M.E2 == 100 ? launch_embed_bwd_cmp<100>(M, D, ti, pos, perm, box, nbrs, T, dG, F4, virial, st)
                       : launch_embed_bwd_cmp<64>(M, D, ti, pos, perm, box, nbrs, T, dG, F4, virial, st);
    if (rc) return rc;
  }
  prof_end(PROF_EMBED_BWD, st);
  return DPB_OK;
}

// Descriptor stage alone (diagnostics): T and G as FP32; the FP16 G of the
// tensor-core kernel is staged in the caller's workspace.
int mixed_descriptors_f32(const DevModel &M, const SysDesc &D, const float *pos, const int32_t *perm,
                          const float *box, const int32_t *nbrs, float *T, float *G, int *err, void *ws,
                          cudaStream_t st) {
  const size_t NG = (size_t)D.N * D.F * M.A * M.E2;
  __half *Gb = reinterpret_cast<__half *>(ws);
  float4 *posS = reinterpret_cast<float4 *>(static_cast<char *>(ws) + al256(NG * 2));
  int rc = launch_pos_sorted(D, pos, perm, posS, st);
  if (rc) return rc;
  rc = mixed_descriptors(M, D, posS, box, nbrs, T, Gb, nullptr, nullptr, err, st);
  if (rc) return rc;
  k_f16_to_f32<<<(unsigned)((NG + 255) / 256), 256, 0, st>>>(Gb, G, NG);
  count_launch();
  DPB_LAUNCH_CHECK();
  return DPB_OK;
}

// Workspace layout of mixed_eval.
struct MixedWs {
  int *err;
  float *T;
  __half *Gb;  // the descriptor G (FP16), the fitting's input
  float *dG;
  __half *dTh;   // dE/dT rows (FP16, scaled per atom)
  float *dTs;    // per-atom inverse scale of dTh
  float4 *posS;
  float4 *rows;  // the forward's compacted neighbour rows (kRowStoreCap per atom)
  int *rcnt;     // their count per block and neighbour type
  float *scratch;
};

static MixedWs mixed_ws(const DevModel &M, size_t NF, void *ws) {
  const int K0 = M.A * M.E2, N2 = n2_of(M);
  char *w = (char *)ws;
  MixedWs o;
  o.err = (int *)w; w += 256;
  o.T = (float *)w; w += al256(NF * 10 * M.E2 * 4);
  o.Gb = (__half *)w; w += al256(NF * K0 * 2);
  o.dG = (float *)w; w += al256(NF * K0 * 4);
  o.dTh = (__half *)w; w += al256(NF * 10 * N2 * 2);
  o.dTs = (float *)w; w += al256(NF * 4);
  o.posS = (float4 *)w; w += al256(NF * 16);
  o.rows = (float4 *)w; w += al256(NF * kRowStoreCap * 16);
  o.rcnt = (int *)w; w += al256(NF * M.ntypes * 4);
  o.scratch = (float *)w;
  return o;
}

int mixed_tune_dT(const DevModel &M, size_t NF, void *ws, cudaStream_t st, int *best) {
  if (M.ngrids > 0 || !M.emb_tuned || !best) return DPB_ERR_UNSUPPORTED;  // these take the FP32 adjoint
  const MixedWs w = mixed_ws(M, NF, ws);
  const __half *dGb = reinterpret_cast<const __half *>(w.dG);
  cudaEvent_t a, b;
  DPB_CUDA_TRY(cudaEventCreate(&a));
  DPB_CUDA_TRY(cudaEventCreate(&b));
  const int cand[3] = {2, 4, 8};
  float tbest = 1e30f;
  *best = 4;
  int rc = DPB_OK;
  for (int c = 0; c < 3 && !rc; ++c) {
    rc = launch_mix_dT(M, NF, w.T, dGb, w.dTh, w.dTs, cand[c], st);  // warm-up (idempotent: dTh from dG, T)
    cudaEventRecord(a, st);
    for (int r = 0; r < 5 && !rc; ++r) rc = launch_mix_dT(M, NF, w.T, dGb, w.dTh, w.dTs, cand[c], st);
    cudaEventRecord(b, st);
    if (cudaEventSynchronize(b) != cudaSuccess) rc = DPB_ERR_CUDA;
    float ms = 0.f;
    cudaEventElapsedTime(&ms, a, b);
    if (!rc && ms < tbest) { tbest = ms; *best = cand[c]; }
  }
  cudaEventDestroy(a);
  cudaEventDestroy(b);
  return rc;
}

// The error word of mixed_eval's workspace, zero on its entry.
int *mixed_err(const DevModel &M, size_t NF, void *ws) { return mixed_ws(M, NF, ws).err; }

int mixed_eval(const DevModel &M, const SysDesc &D, const float *pos, const int32_t *perm, const float *box,
               const int32_t *nbrs, double *energy, float *Eatom, ForceSum *F4, double *virial, void *ws,
               cudaStream_t st, int dT_warps, FitShape fit) {
  const size_t NF = (size_t)D.N * D.F;
  const MixedWs mw = mixed_ws(M, NF, ws);
  int *err = mw.err;
  float *T = mw.T, *dG = mw.dG, *scratch = mw.scratch;
  __half *Gb = mw.Gb;
  float4 *posS = mw.posS;
  if (M.ngrids > 0 || !M.emb_tuned)
    return mixed_eval_compressed(M, D, pos, perm, box, nbrs, energy, Eatom, F4, virial, T, Gb, dG, scratch, err,
                                 fit, st);
  int rc = launch_pos_sorted(D, pos, perm, posS, st);
  if (rc) return rc;
  rc = mixed_descriptors(M, D, posS, box, nbrs, T, Gb, mw.rows, mw.rcnt, err, st);
  if (rc) return rc;
  prof_begin(PROF_MIXED_FIT, st);
  __half *dGb = reinterpret_cast<__half *>(dG);  // dE/dG in FP16 times fit_dgsc (the dE/dT input)
  rc = launch_mix_fit_any<__half>(M, D, Gb, dGb, scratch, Eatom, energy, err, fit, st);
  prof_end(PROF_MIXED_FIT, st);
  if (rc) return rc;
  prof_begin(PROF_MIXED_DT, st);
  rc = launch_mix_dT(M, NF, T, dGb, mw.dTh, mw.dTs, dT_warps, st);
  if (rc) return rc;
  prof_end(PROF_MIXED_DT, st);
  prof_begin(PROF_MIXED_EMBED_BWD, st);
  rc = (M.E2 == 100) ? launch_mix_embed_bwd<25, 50, 100>(M, D, posS, box, nbrs, mw.dTh, mw.dTs, mw.rows, mw.rcnt, F4,
                                                         virial, err, st)
                     : launch_mix_embed_bwd<32, 32, 64>(M, D, posS, box, nbrs, mw.dTh, mw.dTs, mw.rows, mw.rcnt, F4,
                                                        virial, err, st);
  if (rc) return rc;
  prof_end(PROF_MIXED_EMBED_BWD, st);
  return DPB_OK;
}

}  // namespace dpb

extern "C" int dpb_selftest_tcgen05(int variant, float *out, int *err, void *stream) {
  if (!out || !err || variant < 0 || variant > 1) return DPB_ERR_INVALID_ARG;
  dpb::k_selftest_umma<<<1, 128, 0, (cudaStream_t)stream>>>(variant, out, err);
  dpb::count_launch();
  return cudaGetLastError() == cudaSuccess ? DPB_OK : DPB_ERR_CUDA;
}

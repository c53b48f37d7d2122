// FP32 embedding on the tensor cores: forward and adjoint of the tuned
// three-layer nets with every GEMM operand split into FP16 hi + lo parts.
//
// A GEMM of FP32 operands is three FP16 MMAs (lo.hi, hi.lo, hi.hi, smallest
// first) into one FP32 accumulator; weights are scaled by a power of two before
// the split, tangents by one that keeps their bound in range, so hi + lo carry
// about 22 significant bits (activations are not scaled: below 1/8 the lo part's
// error is 3e-8).  tanh, residuals, env rows, the contraction T = R~^T h2 and its
// adjoint stay FP32 multiply-adds.  Against float64 forces, atom energies and
// virials are closer than with the multiply-add form that this replaced (999 to
// 98,304 atoms: the nearest image d - L rint(d / L) also loses less of the
// displacement than the two-step remainder did; and in boxes of several images,
// where the displacement is the same, forces 1.0e-6 to 1.3e-6 against 1.3e-6 to
// 1.6e-6).  A frame's energy carries an error of one sign per model, up to 4e-7 of
// sum |E_atom| (1.6e-7 over 16 random models, 1.3e-7 before): truncated accumulations
// and the activations' 22 bits move every row's h the same way.
//
// Why this split: per neighbour row the nets cost 6,250 multiply-adds forward
// and 12,500 in the adjoint, which the FP32 pipe (128 per clock and SM) cannot
// do in less than 5 ms at 98,304 atoms; on the tensor cores they take a
// fraction of that, and what bounds the kernels is the issue of the 175 tanh
// of a row and of the FP32 contraction.
//
// A operands live in TMEM (written by the epilogues with tcgen05.st, two K
// elements per 32-bit column), so shared memory holds only the resident net
// and two CTAs fit on an SM; TMEM per CTA: 128 accumulator columns, 128 for
// the A operands (forward: 64, the other 64 keep T).
#include "rows.cuh"
#include <algorithm>
#include <cmath>
#include <type_traits>
#include <vector>

namespace dpb {

using tc::f2;

constexpr int kSplitThreads = 256;  // two threads per row
constexpr int kSplitRowCap = 128 + kSplitThreads;

template <int E0, int E1, int E2>
struct SplitDims {
  static constexpr int K1 = (E0 + 15) / 16 * 16, N1 = (E1 + 15) / 16 * 16, K2 = (E1 + 15) / 16 * 16;
  static constexpr int Z1 = E1 / E0, Z2 = E2 / E1;
  // half 0 of a row's two threads owns h1 columns [0, S1) and h2 columns [0,
  // S2), half 1 the rest (their residual sources h[c / Z] included)
  static constexpr int S1 = (E1 / 2) / 8 * 8, S2 = S1 * Z2;
  // layer 2 runs in two passes; pass p covers columns [p P0, p P0 + P0) of
  // half 0 at accumulator columns [0, P0) and [S2 + p P1, S2 + p P1 + P1) of
  // half 1 at [HP, HP + P1); the weight image stores its rows in that order
  static constexpr int P0 = S2 / 2, P1 = (E2 - S2) / 2;
  static constexpr int HP = ((P0 > P1 ? P0 : P1) + 7) / 8 * 8, NP = 2 * HP;
  static constexpr int W1B = N1 * K1 * 2, W2B = NP * K2 * 2;  // one hi (or lo) tile
  static constexpr int IMG = 2 * W1B + 4 * W2B;               // W1 hi, lo; per pass W2 hi, lo
  // w0, w0 times the tangent scale, b0, b1, b2 (pass order), unscale of W1,
  // W2, of the tangents
  static constexpr int O_W0 = 0, O_W0T = 32, O_B0 = 64, O_B1 = 96, O_B2 = 96 + N1, O_SC = O_B2 + 2 * NP,
                       SMALL = O_SC + 4;
  static constexpr int A0C = K1 / 2;  // A0 operand columns [0, A0C) belong to half 0
  static constexpr int H0LO1 = (A0C < S1 / Z1 ? A0C : S1 / Z1) / 2 * 2;
  static constexpr int H0N = K1 / 2 > E0 - H0LO1 ? K1 / 2 : (E0 - H0LO1 + 1) / 2 * 2;
  static constexpr int H1N = S1 > (E1 - S1 + 1) / 2 * 2 ? S1 : (E1 - S1 + 1) / 2 * 2;
  static_assert(Z1 * E0 == E1 && Z2 * E1 == E2 && Z1 <= 2 && Z2 <= 2, "residual ratios 1 or 2");
  static_assert(K1 <= 32 && N1 <= 64 && NP <= 64 && E0 <= 32, "tile widths");
  static_assert(S2 % 2 == 0 && P0 % (2 * Z2) == 0 && P1 % 2 == 0 && (E2 - S2) % 2 == 0, "pass split");
  static_assert(S1 / Z1 <= A0C && (A0C % 8) == 0, "half 0 computes its residual sources");
  static_assert(E2 % 4 == 0, "columns in quads");
};

// TMEM columns of a CTA (256): accumulators, A operands, and (forward) T
constexpr uint32_t kTmX = 0, kTmY = 128, kTmT = 192;

// Host side: hi + lo parts of one layer's weights w (K x N, row-major) times
// sc.  lo keeps 11 bits of the remainder, so about a quarter of the weights are
// off by one unit of their last place; fixed weights make that a systematic
// error of every row, the largest one of the whole split form (energies
// 4e-7 relative).  Each inexact lo is therefore rounded up or down, largest
// effect first, so that the errors of an output column cancel along the layer's
// inputs at nodes of s~ over its range (H, J x K): energies 2e-7, as with exact
// weights.
static void split_weights(const float *w, int K, int N, float sc, const std::vector<double> &H, int J,
                          std::vector<__half> &hi, std::vector<__half> &lo) {
  hi.resize((size_t)K * N);
  lo.resize((size_t)K * N);
  std::vector<double> reach(K, 0.0);
  for (int j = 0; j < J; ++j)
    for (int k = 0; k < K; ++k) reach[k] = fmax(reach[k], fabs(H[(size_t)j * K + k]));
  struct Item {
    int k;
    __half other;
    double d0, d1, key;
  };
  std::vector<Item> items;
  std::vector<double> e(J);
  for (int n = 0; n < N; ++n) {
    items.clear();
    for (int k = 0; k < K; ++k) {
      const float v = w[(size_t)k * N + n] * sc;
      const __half h = __float2half_rn(v);
      const float r = v - __half2float(h);  // exact
      const __half l = __float2half_rn(r);
      hi[(size_t)k * N + n] = h;
      lo[(size_t)k * N + n] = l;
      const double d0 = (double)__half2float(l) - (double)r;
      if (d0 == 0.0 || !std::isfinite(d0)) continue;
      const __half o = d0 > 0.0 ? __float2half_rd(r) : __float2half_ru(r);
      const double d1 = (double)__half2float(o) - (double)r;
      items.push_back({k, o, d0, d1, fmax(fabs(d0), fabs(d1)) * reach[k]});
    }
    std::sort(items.begin(), items.end(), [](const Item &a, const Item &b) { return a.key > b.key; });
    std::fill(e.begin(), e.end(), 0.0);
    for (const Item &it : items) {
      double q0 = 0.0, q1 = 0.0;
      for (int j = 0; j < J; ++j) {
        const double h = H[(size_t)j * K + it.k], a = e[j] + it.d0 * h, b = e[j] + it.d1 * h;
        q0 += a * a;
        q1 += b * b;
      }
      const double d = q1 < q0 ? it.d1 : it.d0;
      if (q1 < q0) lo[(size_t)it.k * N + n] = it.other;
      for (int j = 0; j < J; ++j) e[j] += d * H[(size_t)j * K + it.k];
    }
  }
}

// Host: the image and the small block of one net (see SplitDims); s~ runs over
// [s_lo, s_hi].
template <int E0, int E1, int E2>
static void split_image(const float *w0, const float *b0, const float *w1, const float *b1, const float *w2,
                        const float *b2, double s_lo, double s_hi, std::vector<char> &img, std::vector<float> &small) {
  using D = SplitDims<E0, E1, E2>;
  img.assign(D::IMG, 0);
  small.assign(D::SMALL, 0.f);
  auto amax = [](const float *a, int n) {
    double m = 0.0;
    for (int i = 0; i < n; ++i) m = fmax(m, fabs((double)a[i]));
    return m;
  };
  const float s1 = pow2_scale_to_2p14(amax(w1, E0 * E1)), s2 = pow2_scale_to_2p14(amax(w2, E1 * E2));
  // the inputs of layers 1 and 2 at nodes of s~
  constexpr int J = 12;
  std::vector<double> H0(J * E0), H1(J * E1);
  for (int j = 0; j < J; ++j) {
    const double s = s_lo + (s_hi - s_lo) * j / (J - 1);
    for (int k = 0; k < E0; ++k) H0[j * E0 + k] = tanh(s * w0[k] + b0[k]);
    for (int n = 0; n < E1; ++n) {
      double z = b1[n];
      for (int k = 0; k < E0; ++k) z += H0[j * E0 + k] * w1[k * E1 + n];
      H1[j * E1 + n] = tanh(z) + H0[j * E0 + n / D::Z1];
    }
  }
  std::vector<__half> h1, l1, h2, l2;
  split_weights(w1, E0, E1, s1, H0, J, h1, l1);
  split_weights(w2, E1, E2, s2, H1, J, h2, l2);
  auto put = [](char *p, int lo_off, uint32_t off, __half h, __half l) {
    *reinterpret_cast<__half *>(p + off) = h;
    *reinterpret_cast<__half *>(p + lo_off + off) = l;
  };
  char *p = img.data();
  for (int n = 0; n < E1; ++n)
    for (int k = 0; k < E0; ++k) put(p, D::W1B, tc::kmajor_off(n, k, D::K1), h1[k * E1 + n], l1[k * E1 + n]);
  p += 2 * D::W1B;
  for (int pass = 0; pass < 2; ++pass, p += 2 * D::W2B)
    for (int n = 0; n < D::NP; ++n) {
      const int h = n / D::HP, i = n - h * D::HP;
      if (i >= (h ? D::P1 : D::P0)) continue;
      const int col = h ? D::S2 + pass * D::P1 + i : pass * D::P0 + i;
      for (int k = 0; k < E1; ++k) put(p, D::W2B, tc::kmajor_off(n, k, D::K2), h2[k * E2 + col], l2[k * E2 + col]);
      small[D::O_B2 + pass * D::NP + n] = b2[col];
    }
  // bound on the tangents dh/ds~ of every layer, scaled into FP16 range:
  // |dh0| <= max |w0|, |dh1| <= |dh0| (1 + max column sum of |W1|)
  double c1 = 0.0;
  for (int n = 0; n < E1; ++n) {
    double s = 0.0;
    for (int k = 0; k < E0; ++k) s += fabs((double)w1[k * E1 + n]);
    c1 = fmax(c1, s);
  }
  const float ts = pow2_scale_to_2p14(amax(w0, E0) * (1.0 + c1));  // layer 2's operand is dh1
  for (int k = 0; k < E0; ++k) {
    small[D::O_W0 + k] = w0[k];
    small[D::O_W0T + k] = w0[k] * ts;
    small[D::O_B0 + k] = b0[k];
  }
  for (int n = 0; n < E1; ++n) small[D::O_B1 + n] = b1[n];
  small[D::O_SC] = 1.f / s1;
  small[D::O_SC + 1] = 1.f / s2;
  small[D::O_SC + 2] = 1.f / ts;
}

void split_net_image(int E2, const float *w0, const float *b0, const float *w1, const float *b1, const float *w2,
                     const float *b2, double s_lo, double s_hi, std::vector<char> &img, std::vector<float> &small) {
  if (E2 == 100) split_image<25, 50, 100>(w0, b0, w1, b1, w2, b2, s_lo, s_hi, img, small);
  else split_image<32, 32, 64>(w0, b0, w1, b1, w2, b2, s_lo, s_hi, img, small);
}

// Asynchronous copy of one net's image and small block into shared memory.
template <int E0, int E1, int E2>
__device__ __forceinline__ void split_load_net(const DevModel &M, int k, char *netb, float *small) {
  using D = SplitDims<E0, E1, E2>;
  static_assert(D::IMG % 16 == 0 && D::SMALL % 4 == 0, "16-byte copies");
  const char *img = M.spl_img[k];
  for (int e = threadIdx.x; e < D::IMG / 16; e += blockDim.x) tc::cp_async16(netb + 16 * e, img + 16 * e);
  const float *sm = M.spl_small[k];
  for (int e = threadIdx.x; e < D::SMALL / 4; e += blockDim.x) tc::cp_async16(small + 4 * e, sm + 4 * e);
  tc::cp_async_commit();
}

// D (+)= A B of split operands: K / 16 steps of the products lo.hi, hi.lo,
// hi.hi; a: TMEM columns of A hi (K / 2 columns) followed by A lo; b: shared
// address of B hi followed (bytes later) by B lo; K-major.
template <int K>
__device__ __forceinline__ void split_mma(uint32_t d, uint32_t a, uint32_t b, uint32_t b_lo, uint32_t idesc) {
#pragma unroll
  for (int p = 0; p < 3; ++p) {
    const uint32_t ap = a + (p == 0 ? K / 2 : 0), bp = b + (p == 1 ? b_lo : 0);
#pragma unroll
    for (int ks = 0; ks < K / 16; ++ks)
      tc::mma_f16kind_ta(d, ap + 8 * ks, tc::make_desc(bp + tc::kmajor_off(0, 16 * ks, K), 128, (K / 8) * 128), idesc,
                         (p > 0 || ks > 0) ? 1u : 0u);
  }
}

// Four pairs (8 operand columns) of one row as hi and lo words.
__device__ __forceinline__ void split8(const f2 (&v)[4], uint32_t (&hi)[4], uint32_t (&lo)[4]) {
#pragma unroll
  for (int i = 0; i < 4; ++i) tc::split_pair(v[i], hi[i], lo[i]);
}

__device__ __forceinline__ float lo_of(f2 p) {
  float a, b;
  tc::upk(p, a, b);
  return a;
}
__device__ __forceinline__ float hi_of(f2 p) {
  float a, b;
  tc::upk(p, a, b);
  return b;
}
// Residual source of the column pair (c, c + 1), c even and relative to the
// first column of src: the pair itself (ratio 1), or column c / 2 twice.
template <int Z>
__device__ __forceinline__ f2 split_res(const f2 *src, int c) {
  if (Z == 1) return src[c >> 1];
  const int k = c >> 1;
  return tc::pk1((k & 1) ? hi_of(src[k >> 1]) : lo_of(src[k >> 1]));
}

// Layer 0 of one half: h0 = tanh(s~ w0 + b0) and, with TAN, the scaled tangent
// (1 - h0^2) w0 ts, in registers from column H0LO (0 or H0LO1) and as A
// operand words in TMEM.
template <int E0, int E1, int E2, int HALF, bool TAN>
__device__ __forceinline__ void split_layer0(float st, const float *sm, uint32_t tY,
                                             f2 (&h0)[SplitDims<E0, E1, E2>::H0N / 2],
                                             f2 (&d0)[SplitDims<E0, E1, E2>::H0N / 2]) {
  using D = SplitDims<E0, E1, E2>;
  constexpr int lo = HALF ? D::H0LO1 : 0, hi = HALF ? E0 : D::A0C;
  const f2 st2 = tc::pk1(st), one = tc::pk1(1.f);
#pragma unroll
  for (int c = lo; c < hi; c += 2) {  // columns past E0: zero weights, tanh(0) = 0
    const f2 w = *reinterpret_cast<const f2 *>(sm + D::O_W0 + c), b = *reinterpret_cast<const f2 *>(sm + D::O_B0 + c);
    const f2 t = tc::tanh_pair(tc::fma2(st2, w, b));
    h0[(c - lo) / 2] = t;
    if (TAN) {
      const f2 wt = *reinterpret_cast<const f2 *>(sm + D::O_W0T + c);
      const f2 nt = tc::mul2(t, tc::pk1(-1.f));
      d0[(c - lo) / 2] = tc::mul2(tc::fma2(nt, t, one), wt);
    }
  }
  const f2 zero = tc::pk1(0.f);
#pragma unroll
  for (int k8 = HALF ? D::A0C : 0; k8 < (HALF ? D::K1 : D::A0C); k8 += 8) {
    f2 v[4];
    uint32_t wh[4], wl[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) v[i] = k8 + 2 * i < hi ? h0[(k8 - lo) / 2 + i] : zero;
    split8(v, wh, wl);
    tc::tmem_st4(tY + k8 / 2, wh);
    tc::tmem_st4(tY + D::K1 / 2 + k8 / 2, wl);
    if (TAN) {
#pragma unroll
      for (int i = 0; i < 4; ++i) v[i] = k8 + 2 * i < hi ? d0[(k8 - lo) / 2 + i] : zero;
      split8(v, wh, wl);
      tc::tmem_st4(tY + D::K1 + k8 / 2, wh);
      tc::tmem_st4(tY + D::K1 + D::K1 / 2 + k8 / 2, wl);
    }
  }
}

// Layer 1 epilogue of one half: h1 = tanh(z1 + b1) + rep(h0), with TAN dh1 =
// (1 - t^2) dz1 + rep(dh0), from the accumulators at tX (tangent at tX + N1),
// kept in registers and written as A operand words at tY.
template <int E0, int E1, int E2, int HALF, bool TAN>
__device__ __forceinline__ void split_layer1(uint32_t tX, uint32_t tY, const float *sm,
                                             const f2 (&h0)[SplitDims<E0, E1, E2>::H0N / 2],
                                             const f2 (&d0)[SplitDims<E0, E1, E2>::H0N / 2],
                                             f2 (&h1)[SplitDims<E0, E1, E2>::H1N / 2],
                                             f2 (&d1)[SplitDims<E0, E1, E2>::H1N / 2]) {
  using D = SplitDims<E0, E1, E2>;
  constexpr int c0 = HALF ? D::S1 : 0, c1 = HALF ? E1 : D::S1, kEnd = HALF ? D::K2 : D::S1;
  constexpr int h0lo = HALF ? D::H0LO1 : 0;
  const f2 us = tc::pk1(sm[D::O_SC]), one = tc::pk1(1.f), zero = tc::pk1(0.f);
#pragma unroll
  for (int g = c0; g < kEnd; g += 8) {
    uint32_t z[8], dz[8];
    if (g < c1) {
      tc::tmem_ld8_issue(tX + g, z);
      if (TAN) tc::tmem_ld8_issue(tX + D::N1 + g, dz);
      tc::tmem_wait();
    }
    f2 hv[4], dv[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int c = g + 2 * i;
      hv[i] = dv[i] = zero;
      if (c < c1) {
        const f2 b = *reinterpret_cast<const f2 *>(sm + D::O_B1 + c);
        const f2 t = tc::tanh_pair(
            tc::fma2(tc::pk(__uint_as_float(z[2 * i]), __uint_as_float(z[2 * i + 1])), us, b));
        hv[i] = tc::add2(t, split_res<D::Z1>(h0, c - h0lo * D::Z1));
        h1[(c - c0) / 2] = hv[i];
        if (TAN) {
          const f2 u = tc::mul2(tc::fma2(tc::mul2(t, tc::pk1(-1.f)), t, one), us);
          dv[i] = tc::fma2(u, tc::pk(__uint_as_float(dz[2 * i]), __uint_as_float(dz[2 * i + 1])),
                           split_res<D::Z1>(d0, c - h0lo * D::Z1));
          d1[(c - c0) / 2] = dv[i];
        }
      }
    }
    uint32_t wh[4], wl[4];
    split8(hv, wh, wl);
    tc::tmem_st4(tY + g / 2, wh);
    tc::tmem_st4(tY + D::K2 / 2 + g / 2, wl);
    if (TAN) {
      split8(dv, wh, wl);
      tc::tmem_st4(tY + D::K2 + g / 2, wh);
      tc::tmem_st4(tY + D::K2 + D::K2 / 2 + g / 2, wl);
    }
  }
}

// Geometry and env row of a stored row (FP32, true divisions).
__device__ __forceinline__ void split_row_env(float4 rb, float rcut, float inv_std, float mean, RowGeom &gm,
                                              float &st, float (&R)[10]) {
  row_geom(make_float3(rb.x, rb.y, rb.z), rcut, gm);
  st = (gm.s - mean) * inv_std;
  const float inv_rp = 1.f / (gm.r + 1e-16f);
  const float xh[3] = {gm.x[0] * inv_rp, gm.x[1] * inv_rp, gm.x[2] * inv_rp};
  env_row(gm.s * inv_std, xh, R);
}

// ---------------------------------------------------------------- forward
// Persistent CTAs over blocks of up to 4 centre atoms (of both centre types in
// one launch).  Rows of one neighbour type are packed into 128-row tiles: layer
// 0 -> A0 -> tcgen05 -> layer 1 -> A1 -> tcgen05 (both passes) -> h2 in shared
// memory, and T[slot][c][w] = sum_rows R[c] h2[w] as FP32 multiply-adds: thread
// (column quad q, channel pair p, row split s) keeps 8 sums in registers for
// the current slot and 8 TMEM words per slot, that only it touches, for the
// totals; the two row splits meet in the block epilogue.  The contraction of
// tile k runs while the first MMA of tile k + 1 is in flight.
template <int E0, int E1, int E2>
struct SplitFwdSmem {
  using D = SplitDims<E0, E1, E2>;
  static constexpr int HS = E2 % 32 ? E2 : E2 + 4;  // h2 row stride (floats): rows r and r + 4 in different banks
  static constexpr int RS = 12;        // env row stride
  static constexpr int net = 0, small = net + D::IMG, h2 = small + (D::SMALL * 4 + 127) / 128 * 128,
                       env = h2 + 128 * HS * 4, rowbuf = env + 128 * RS * 4, stash = rowbuf + kSplitRowCap * 16,
                       total = stash + 8 * kSplitThreads * 4;
};

template <int E0, int E1, int E2>
__global__ void __launch_bounds__(kSplitThreads, 2) k_split_fwd(DevModel M, SysDesc D, int ba,
                                                               const float4 *__restrict__ posS,
                                                               const float *__restrict__ box,
                                                               const int32_t *__restrict__ nbrs,
                                                               const float4 *__restrict__ rows_g,
                                                               const int *__restrict__ rcnt, float *__restrict__ Tout,
                                                               float *__restrict__ Gout, float *__restrict__ gmax,
                                                               int *__restrict__ err) {
  using SD = SplitDims<E0, E1, E2>;
  using SM = SplitFwdSmem<E0, E1, E2>;
  extern __shared__ __align__(1024) char smem[];
  char *netb = smem + SM::net;
  float *sm = reinterpret_cast<float *>(smem + SM::small);
  float *h2s = reinterpret_cast<float *>(smem + SM::h2), *envs = reinterpret_cast<float *>(smem + SM::env);
  float4 *rowbuf = reinterpret_cast<float4 *>(smem + SM::rowbuf);
  float *stash = reinterpret_cast<float *>(smem + SM::stash);  // running sums, [8][thread]
  __shared__ int wcnt[kSplitThreads / 32];
  __shared__ int seg_s[5];  // first row of each slot in the staged tile
  __shared__ float3 ri_s[kBlkAtoms];
  __shared__ int gmax_s[4];  // largest |G| per slot (float bits)
  __shared__ __align__(8) uint64_t mbar;
  __shared__ uint32_t tbase_s;
  const int tid = threadIdx.x, warp = tc::warp_index();
  const int row = tid & 127, half = tid >> 7;
  if (tid == 0) tc::mbar_init(&mbar, 1);
  if (warp == 0) tc::tmem_alloc(&tbase_s, 256);
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tbase = tbase_s, lane_off = (uint32_t)((warp & 3) * 32) << 16;
  const uint32_t tX = tbase + kTmX, tY = tbase + kTmY;
  const uint32_t tT = tbase + kTmT + lane_off + (warp >> 2) * 32;  // this thread's T words, 8 per slot
  uint32_t ph = 0;
  bool ok = true;
  const uint32_t idesc1 = tc::idesc_f16(128, SD::N1, 0, 0), idesc2 = tc::idesc_f16(128, SD::NP, 0, 0);
  const uint32_t w1_u = tc::smem_u32(netb), w2_u = w1_u + 2 * SD::W1B;
  // the contraction's role: quad q, channel pair p, row split s
  constexpr int NCT = (E2 / 4) * 10;
  const int cs = tid & 1, cp = (tid >> 1) % 5, cq = (tid >> 1) / 5;
  const bool crole = tid < NCT;
  const int nblk = blocks_total(D, ba);
  int loaded_net = -1;

  for (int blk = blockIdx.x; blk < nblk && ok; blk += gridDim.x) {
    const BlkPos bp = block_pos(D, ba, blk);
    const int ti = bp.ti, nb = bp.nb, f = bp.f;
    const size_t g0 = bp.g0, frame_base = (size_t)f * D.N;
    const float inv_std = M.inv_std[ti], mean = M.mean[ti];
    if (blk + (int)gridDim.x < nblk) {  // the next block's neighbour rows
      const BlkPos bn = block_pos(D, ba, blk + gridDim.x);
      if (rows_g != nullptr && D.S <= kRowStoreCap)
        prefetch_range_l2(rows_g + bn.g0 * kRowStoreCap, (size_t)bn.nb * D.S * 16);
      else prefetch_range_l2(nbrs + bn.g0 * D.S, (size_t)bn.nb * D.S * 4);
    }
    const int bs = box_slot(D, g0, f);
    const float3 L = make_float3(box[bs * 3], box[bs * 3 + 1], box[bs * 3 + 2]);
    const int3 ni = image_range(L, M.rcut);
    const int nim = (2 * ni.x + 1) * (2 * ni.y + 1) * (2 * ni.z + 1);
    const bool stream = row_store_covers(D, rows_g, nim);
    if (tid < nb) {
      const float4 q = posS[g0 + tid];
      ri_s[tid] = make_float3(q.x, q.y, q.z);
    }
    __syncthreads();
    unsigned touched = 0;    // slots with a sum in TMEM (uniform)
    int staged = -1;         // neighbour type of the tile in h2 / env rows that waits for its contraction
    int open_slot = -1, open_tj = -1, open_off = 0;  // the slot whose sum is still running, its type and rows so far
    // adds the running sum to its slot's total
    auto close = [&]() {
      if (open_slot < 0) return;
      uint32_t w[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) w[i] = __float_as_uint(stash[i * kSplitThreads + tid]);
      if (touched >> open_slot & 1u) {
        uint32_t o[8];
        tc::tmem_ld8_issue(tT + 8 * open_slot, o);
        tc::tmem_wait();
#pragma unroll
        for (int i = 0; i < 8; ++i) w[i] = __float_as_uint(__uint_as_float(w[i]) + __uint_as_float(o[i]));
      }
      tc::tmem_st8(tT + 8 * open_slot, w);
      tc::tmem_wait_st();
      touched |= 1u << open_slot;
      open_slot = -1;
    };
    // A slot's rows of one neighbour type are summed in list order, four rows
    // in turn per row split, across tile boundaries: the result does not depend
    // on how the rows fall into tiles or blocks, so a frame gives the same bits
    // alone and in a packed batch.
    auto contract = [&]() {
#pragma unroll 1
      for (int sl = 0; sl < nb; ++sl) {
        const int b = seg_s[sl], e = seg_s[sl + 1];
        if (b >= e) continue;
        const bool cont = open_slot == sl && open_tj == staged;
        if (!cont) close();
        const int off = cont ? open_off : 0;
        f2 s00 = tc::pk1(0.f), s01 = s00, s10 = s00, s11 = s00;
        if (crole) {
          float *stp = stash + tid;
          if (cont) {
            s00 = tc::pk(stp[0], stp[kSplitThreads]);
            s01 = tc::pk(stp[2 * kSplitThreads], stp[3 * kSplitThreads]);
            s10 = tc::pk(stp[4 * kSplitThreads], stp[5 * kSplitThreads]);
            s11 = tc::pk(stp[6 * kSplitThreads], stp[7 * kSplitThreads]);
          }
          const float *hq = h2s + 4 * cq, *rp = envs + 2 * cp;
          auto rowfma = [&](int r) {
            const float4 h = *reinterpret_cast<const float4 *>(hq + r * SM::HS);
            const float2 R = *reinterpret_cast<const float2 *>(rp + r * SM::RS);
            const f2 ha = tc::pk(h.x, h.y), hb = tc::pk(h.z, h.w), r0 = tc::pk1(R.x), r1 = tc::pk1(R.y);
            s00 = tc::fma2(ha, r0, s00);
            s01 = tc::fma2(hb, r0, s01);
            s10 = tc::fma2(ha, r1, s10);
            s11 = tc::fma2(hb, r1, s11);
          };
          for (int k8 = b - (off & 7); k8 < e; k8 += 8) {  // rows k8 + 4 cs + 0..3 of [b, e)
            const int r0 = k8 + 4 * cs;
            if (r0 >= b && r0 + 4 <= e) {
#pragma unroll
              for (int j = 0; j < 4; ++j) rowfma(r0 + j);
            } else {
              for (int r = max(r0, b); r < min(r0 + 4, e); ++r) rowfma(r);
            }
          }
          float v0, v1;
          tc::upk(s00, v0, v1); stp[0] = v0; stp[kSplitThreads] = v1;
          tc::upk(s01, v0, v1); stp[2 * kSplitThreads] = v0; stp[3 * kSplitThreads] = v1;
          tc::upk(s10, v0, v1); stp[4 * kSplitThreads] = v0; stp[5 * kSplitThreads] = v1;
          tc::upk(s11, v0, v1); stp[6 * kSplitThreads] = v0; stp[7 * kSplitThreads] = v1;
        }
        open_slot = sl;
        open_tj = staged;
        open_off = off + e - b;
      }
      staged = -1;
    };
    int rowstart = 0, rowcount = 0;
    // start with the resident net's type (the sum of two types commutes; more keep their order)
    const int tj0 = (D.ntypes == 2 && loaded_net >= 0 && loaded_net / M.ntypes == ti) ? loaded_net - ti * M.ntypes : 0;
    for (int tt = 0; tt < D.ntypes && ok; ++tt) {
      const int tj = (tj0 + tt) % D.ntypes;
      const int per_atom = D.sel[tj] * nim, total = nb * per_atom;
      const int knet = ti * M.ntypes + tj;
      const float4 *rsrc = stream ? rows_g + g0 * kRowStoreCap + (size_t)nb * D.col[tj] : nullptr;
      const int nsrc = stream ? rcnt[g0 * M.ntypes + tj] : total;
      for (int base = 0; base < nsrc + kSplitThreads && ok; base += kSplitThreads) {
        const bool flush = base >= nsrc;
        if (!flush) {
          if (stream) mix_stream_round<1>(rsrc, base, nsrc, rowbuf, rowstart, rowcount);
          else
            mix_compact_round<1>(D, M, tj, base, total, per_atom, nim, ni, L, g0, frame_base, ri_s, posS, nbrs, rowbuf,
                                 wcnt, rowstart, rowcount);
        }
        while (rowcount - rowstart >= 128 || (flush && rowcount > rowstart)) {
          const int nrows = min(rowcount - rowstart, 128);
          if (loaded_net != knet) {
            __syncthreads();
            split_load_net<E0, E1, E2>(M, knet, netb, sm);
            loaded_net = knet;
          }
          const bool act = row < nrows;
          const float4 rv = act ? rowbuf[rowstart + row] : make_float4(100.f, 100.f, 100.f, 0.f);
          const int slot = act ? (__float_as_int(rv.w) & 7) : nb;
          const int pslot = row == 0 ? -1 : (row - 1 < nrows ? (__float_as_int(rowbuf[rowstart + row - 1].w) & 7) : nb);
          RowGeom gm;
          float st, R[10];
          split_row_env(rv, M.rcut, inv_std, mean, gm, st, R);
          tc::cp_async_wait<0>();
          __syncthreads();  // net image visible; rowbuf read by every thread
          f2 h1[SD::H1N / 2];
          {
            f2 h0[SD::H0N / 2];
            if (half == 0) split_layer0<E0, E1, E2, 0, false>(st, sm, tY + lane_off, h0, h0);
            else split_layer0<E0, E1, E2, 1, false>(st, sm, tY + lane_off, h0, h0);
            tc::tmem_wait_st();
            tc::fence_proxy_async();  // the net image, copied with cp.async
            tc::fence_before_sync();
            __syncthreads();
            if (warp == 0 && tc::elect_one()) {
              tc::fence_after_sync();
              split_mma<SD::K1>(tX, tY, w1_u, SD::W1B, idesc1);
              tc::commit(&mbar);
            }
            if (staged >= 0) contract();
            MIX_WAIT();
            if (!ok) break;
            if (half == 0) split_layer1<E0, E1, E2, 0, false>(tX + lane_off, tY + lane_off, sm, h0, h0, h1, h1);
            else split_layer1<E0, E1, E2, 1, false>(tX + lane_off, tY + lane_off, sm, h0, h0, h1, h1);
          }
          tc::tmem_wait_st();
          tc::fence_before_sync();
          __syncthreads();
          if (warp == 0 && tc::elect_one()) {
            tc::fence_after_sync();
            split_mma<SD::K2>(tX, tY, w2_u, SD::W2B, idesc2);
            split_mma<SD::K2>(tX + SD::NP, tY, w2_u + 2 * SD::W2B, SD::W2B, idesc2);
            tc::commit(&mbar);
          }
          // the env rows and slot ranges of this tile (the previous tile's are contracted)
          if (half == 0) {
#pragma unroll
            for (int c = 0; c < 10; c += 2)
              *reinterpret_cast<float2 *>(envs + row * SM::RS + c) = make_float2(R[c], R[c + 1]);
            for (int s = pslot + 1; s <= slot; ++s) seg_s[s] = row;
            if (row == 127)
              for (int s = slot + 1; s <= nb; ++s) seg_s[s] = 128;
          }
          MIX_WAIT();
          if (!ok) break;
          // layer 2: h2 = tanh(z2 + b2) + rep(h1) to shared memory
          {
            const f2 us = tc::pk1(sm[SD::O_SC + 1]);
            float *hrow = h2s + row * SM::HS;
            auto epi2 = [&](auto HALF) {
              constexpr int H = decltype(HALF)::value, P = H ? SD::P1 : SD::P0;
#pragma unroll
              for (int pass = 0; pass < 2; ++pass)
#pragma unroll
                for (int g = 0; g < P; g += 8) {
                  uint32_t z[8];
                  tc::tmem_ld8_issue(tX + lane_off + pass * SD::NP + H * SD::HP + g, z);
                  tc::tmem_wait();
#pragma unroll
                  for (int i = 0; i < 8; i += 2)
                    if (g + i < P) {
                      const int pc = pass * P + g + i;  // column within the half
                      const f2 b = *reinterpret_cast<const f2 *>(sm + SD::O_B2 + pass * SD::NP + H * SD::HP + g + i);
                      const f2 t =
                          tc::tanh_pair(tc::fma2(tc::pk(__uint_as_float(z[i]), __uint_as_float(z[i + 1])), us, b));
                      *reinterpret_cast<f2 *>(hrow + H * SD::S2 + pc) = tc::add2(t, split_res<SD::Z2>(h1, pc));
                    }
                }
            };
            if (half == 0) epi2(std::integral_constant<int, 0>());
            else epi2(std::integral_constant<int, 1>());
          }
          tc::fence_before_sync();
          staged = tj;
          rowstart += nrows;
          __syncthreads();
        }
      }
    }
    if (!ok) break;
    if (staged >= 0) contract();
    close();
    __syncthreads();  // the contraction has read h2
    // ---- block epilogue: X = T / Nnbrs [slot][c][w] over the h2 region, T out, G out
    float *Xs = h2s;
#pragma unroll 1
    for (int sl = 0; sl < nb; ++sl) {
      uint32_t w[8];
      if (touched >> sl & 1u) {
        tc::tmem_ld8_issue(tT + 8 * sl, w);
        tc::tmem_wait();
      } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) w[i] = 0u;
      }
#pragma unroll
      for (int i = 0; i < 8; ++i)  // the two row splits
        w[i] = __float_as_uint(__uint_as_float(w[i]) + __shfl_xor_sync(0xffffffffu, __uint_as_float(w[i]), 1));
      if (crole && cs == 0) {
#pragma unroll
        for (int ch = 0; ch < 2; ++ch)
          *reinterpret_cast<float4 *>(Xs + (sl * 10 + 2 * cp + ch) * E2 + 4 * cq) =
              make_float4(__uint_as_float(w[4 * ch]) * M.inv_nnbrs, __uint_as_float(w[4 * ch + 1]) * M.inv_nnbrs,
                          __uint_as_float(w[4 * ch + 2]) * M.inv_nnbrs, __uint_as_float(w[4 * ch + 3]) * M.inv_nnbrs);
      }
    }
    __syncthreads();
    {
      const int n4 = nb * 10 * E2 / 4;
      float4 *dst = reinterpret_cast<float4 *>(Tout + g0 * 10 * E2);
      for (int e = tid; e < n4; e += kSplitThreads) dst[e] = reinterpret_cast<const float4 *>(Xs)[e];
    }
    // G[a][w] = sum_c Q[c][a] X[c][w], X = T + Tbias on channel 0 (dpmodel.py:74-78);
    // Q[slot][a][12] staged behind X
    const int A = M.A;
    float *Qs = Xs + 4 * 10 * E2;
    if (tid < 4) gmax_s[tid] = 0;
    for (int e = tid; e < nb * 160; e += kSplitThreads) {
      const int slot = e / 160, aa = (e - slot * 160) / 10, c = e - slot * 160 - aa * 10;
      if (aa < A) {
        const float *X = Xs + slot * 10 * E2;
        float q;
        if (c < 4) {
          q = X[c * E2 + aa] + (c == 0 ? M.tbias[aa] : 0.f);
        } else {
          const float y1 = X[E2 + A + aa], y2 = X[2 * E2 + A + aa], y3 = X[3 * E2 + A + aa];
          const float b6[6] = {y1 * y1, y2 * y2, y3 * y3, kSqrt2 * y1 * y3, kSqrt2 * y2 * y1, kSqrt2 * y3 * y2};
          q = b6[c - 4] + X[c * E2 + A + aa];
        }
        Qs[(slot * 16 + aa) * 12 + c] = q;
      }
    }
    __syncthreads();
    for (int pr = tid; pr < nb * (E2 / 2); pr += kSplitThreads) {
      const int slot = pr / (E2 / 2), w = 2 * (pr - slot * (E2 / 2));
      f2 x[10];
#pragma unroll
      for (int c = 0; c < 10; ++c) x[c] = *reinterpret_cast<const f2 *>(Xs + (slot * 10 + c) * E2 + w);
      x[0] = tc::add2(x[0], tc::pk(M.tbias[w], M.tbias[w + 1]));
      const float *Q = Qs + slot * 16 * 12;
      float *Gs = Gout + (g0 + slot) * (size_t)A * E2 + w;
      float gm = 0.f;
      for (int aa = 0; aa < A; ++aa, Q += 12) {
        const float4 qa = *reinterpret_cast<const float4 *>(Q), qb = *reinterpret_cast<const float4 *>(Q + 4);
        const float2 qc = *reinterpret_cast<const float2 *>(Q + 8);
        f2 v = tc::mul2(x[0], tc::pk1(qa.x));
        v = tc::fma2(x[1], tc::pk1(qa.y), v);
        v = tc::fma2(x[2], tc::pk1(qa.z), v);
        v = tc::fma2(x[3], tc::pk1(qa.w), v);
        v = tc::fma2(x[4], tc::pk1(qb.x), v);
        v = tc::fma2(x[5], tc::pk1(qb.y), v);
        v = tc::fma2(x[6], tc::pk1(qb.z), v);
        v = tc::fma2(x[7], tc::pk1(qb.w), v);
        v = tc::fma2(x[8], tc::pk1(qc.x), v);
        v = tc::fma2(x[9], tc::pk1(qc.y), v);
        *reinterpret_cast<f2 *>(Gs + (size_t)aa * E2) = v;
        gm = fmaxf(gm, fmaxf(fabsf(lo_of(v)), fabsf(hi_of(v))));
      }
      atomicMax(&gmax_s[slot], __float_as_int(gm));  // gm >= 0: the bits order as the values
    }
    __syncthreads();
    if (gmax && tid < nb) gmax[g0 + tid] = __int_as_float(gmax_s[tid]);
  }
  if (!ok) {
    if (tid == 0) atomicOr(err, 1);  // a tensor-core wait gave up (k_finalize)
    tc::mbar_wait(&mbar, ph);
  }
  tc::cp_async_wait<0>();
  tc::fence_before_sync();
  __syncthreads();
  if (warp == 0) tc::tmem_dealloc(tbase, 256);
}

// ---------------------------------------------------------------- dE/dT
// Adjoint of the descriptor, one warp per atom: from dE/dG (A x E2) and T (10 x
// E2), dQ[c][a] = sum_w X[c][w] dG[a][w], dX[c][w] = sum_a Q[c][a] dG[a][w] plus
// the Q -> X terms at w < 2A; dE/dT = dX / Nnbrs overwrites T.  FP32
// multiply-adds on packed pairs; lanes own column quads (dX) and (a, channel
// half) pairs (dQ).  The next atom's rows are copied while this one's products run
// (with each warp's copies and products in turn, twice the warps per SM: 419 us for
// 98,304 atoms, 381 us now; its memory traffic takes 215 us.)
template <int E2>
struct SplitDtSmem {
  static constexpr int XS = E2, DS = E2 + 4;  // dE/dG rows padded: 16 rows in different banks
  static constexpr int buf = 10 * XS + 16 * DS;
  static constexpr int floats = 2 * buf + 16 * 12 + 160 + 48;
};

constexpr int kSplitDtCtas = 2;  // per SM, by shared memory
template <int E2>
__global__ void __launch_bounds__(128) k_split_dT(DevModel M, int NF, float *__restrict__ T,
                                                 const float *__restrict__ dG) {
  using SM = SplitDtSmem<E2>;
  extern __shared__ __align__(16) float dts[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float *buf = dts + warp * SM::floats, *Q = buf + 2 * SM::buf, *dQ = Q + 16 * 12, *ys = dQ + 160;
  const int A = M.A;
  const size_t stride = (size_t)gridDim.x * 4;
  auto copy = [&](size_t g, float *X) {
    const float *Tg = T + g * 10 * E2, *Gg = dG + g * (size_t)A * E2;
    for (int e = lane; e < 10 * E2 / 4; e += 32) tc::cp_async16(X + 4 * e, Tg + 4 * e);
    for (int e = lane; e < A * (E2 / 4); e += 32) {
      const int a = e / (E2 / 4), w = 4 * (e - a * (E2 / 4));
      tc::cp_async16(X + 10 * SM::XS + a * SM::DS + w, Gg + 4 * e);
    }
  };
  const float4 tb = lane < E2 / 4 ? make_float4(M.tbias[4 * lane], M.tbias[4 * lane + 1], M.tbias[4 * lane + 2],
                                                M.tbias[4 * lane + 3])
                                  : make_float4(0.f, 0.f, 0.f, 0.f);
  size_t g = (size_t)blockIdx.x * 4 + warp;
  if (g < (size_t)NF) copy(g, buf);
  tc::cp_async_commit();
  for (int it = 0; g < (size_t)NF; g += stride, ++it) {
    float *X = buf + (it & 1) * SM::buf, *Dg = X + 10 * SM::XS, *Tg = T + g * 10 * E2;
    if (g + stride < (size_t)NF) copy(g + stride, buf + ((it & 1) ^ 1) * SM::buf);
    tc::cp_async_commit();
    tc::cp_async_wait<1>();
    __syncwarp();
    if (lane < E2 / 4) {  // Tbias on channel 0
      float4 t = *reinterpret_cast<float4 *>(X + 4 * lane);
      t.x += tb.x; t.y += tb.y; t.z += tb.z; t.w += tb.w;
      *reinterpret_cast<float4 *>(X + 4 * lane) = t;
    }
    __syncwarp();
    if (lane < A) {  // Q[a][c] and y_k[a]
      const float y1 = X[E2 + A + lane], y2 = X[2 * E2 + A + lane], y3 = X[3 * E2 + A + lane];
      float q[10];
#pragma unroll
      for (int c = 0; c < 4; ++c) q[c] = X[c * E2 + lane];
      const float b6[6] = {y1 * y1, y2 * y2, y3 * y3, kSqrt2 * y1 * y3, kSqrt2 * y2 * y1, kSqrt2 * y3 * y2};
#pragma unroll
      for (int m = 0; m < 6; ++m) q[4 + m] = b6[m] + X[(4 + m) * E2 + A + lane];
#pragma unroll
      for (int c = 0; c < 10; ++c) Q[lane * 12 + c] = q[c];
      ys[lane] = y1;
      ys[16 + lane] = y2;
      ys[32 + lane] = y3;
    }
    {  // dQ: lane = (a, channels 5 h .. 5 h + 4)
      const int a = lane & 15, h = lane >> 4;
      f2 s[5];
#pragma unroll
      for (int c = 0; c < 5; ++c) s[c] = tc::pk1(0.f);
      if (a < A)
        for (int w = 0; w < E2; w += 4) {
          const float4 d = *reinterpret_cast<const float4 *>(Dg + a * SM::DS + w);
          const f2 da = tc::pk(d.x, d.y), db = tc::pk(d.z, d.w);
#pragma unroll
          for (int c = 0; c < 5; ++c) {
            const float4 x = *reinterpret_cast<const float4 *>(X + (5 * h + c) * SM::XS + w);
            s[c] = tc::fma2(tc::pk(x.x, x.y), da, s[c]);
            s[c] = tc::fma2(tc::pk(x.z, x.w), db, s[c]);
          }
        }
#pragma unroll
      for (int c = 0; c < 5; ++c) dQ[(5 * h + c) * 16 + a] = lo_of(s[c]) + hi_of(s[c]);
    }
    __syncwarp();
    if (lane < E2 / 4) {
      f2 x[10][2];
#pragma unroll
      for (int c = 0; c < 10; ++c) x[c][0] = x[c][1] = tc::pk1(0.f);
      for (int a = 0; a < A; ++a) {
        const float4 d = *reinterpret_cast<const float4 *>(Dg + a * SM::DS + 4 * lane);
        const f2 da = tc::pk(d.x, d.y), db = tc::pk(d.z, d.w);
        const float *q = Q + a * 12;
#pragma unroll
        for (int c = 0; c < 10; ++c) {
          const f2 qc = tc::pk1(q[c]);
          x[c][0] = tc::fma2(da, qc, x[c][0]);
          x[c][1] = tc::fma2(db, qc, x[c][1]);
        }
      }
      float v[10][4];
#pragma unroll
      for (int c = 0; c < 10; ++c) {
        tc::upk(x[c][0], v[c][0], v[c][1]);
        tc::upk(x[c][1], v[c][2], v[c][3]);
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) {  // contributions through Q at w < 2A
        const int w = 4 * lane + i;
        if (w < A) {
#pragma unroll
          for (int c = 0; c < 4; ++c) v[c][i] += dQ[c * 16 + w];
        } else if (w < 2 * A) {
          const int aa = w - A;
          float d2[6];
#pragma unroll
          for (int m = 0; m < 6; ++m) d2[m] = dQ[(4 + m) * 16 + aa];
          const float y1 = ys[aa], y2 = ys[16 + aa], y3 = ys[32 + aa];
#pragma unroll
          for (int m = 0; m < 6; ++m) v[4 + m][i] += d2[m];
          v[1][i] += 2.f * y1 * d2[0] + kSqrt2 * y3 * d2[3] + kSqrt2 * y2 * d2[4];
          v[2][i] += 2.f * y2 * d2[1] + kSqrt2 * y1 * d2[4] + kSqrt2 * y3 * d2[5];
          v[3][i] += 2.f * y3 * d2[2] + kSqrt2 * y1 * d2[3] + kSqrt2 * y2 * d2[5];
        }
      }
#pragma unroll
      for (int c = 0; c < 10; ++c)
        reinterpret_cast<float4 *>(Tg + c * E2)[lane] =
            make_float4(v[c][0] * M.inv_nnbrs, v[c][1] * M.inv_nnbrs, v[c][2] * M.inv_nnbrs, v[c][3] * M.inv_nnbrs);
    }
    __syncwarp();
  }
}

// ---------------------------------------------------------------- adjoint
// The rows are recomputed with their tangent along s~ (forward mode), value and
// tangent operands side by side in TMEM; layer 2 in two passes of 64
// accumulator columns each for value and tangent.  Each thread multiplies its
// columns of h2 and dh2 by dE/dT of the row's slot (FP32, dT[slot][w][12] in
// shared memory): u = dE/dR~ and v, dE/ds~ = R~ . v; half 1 hands its partial
// sums to half 0, which finishes the row: env adjoint, neighbour force scatter,
// virial, and the centre force by a segmented warp sum.
template <int E0, int E1, int E2>
struct SplitBwdSmem {
  using D = SplitDims<E0, E1, E2>;
  static constexpr int net = 0, small = net + D::IMG, dT = small + (D::SMALL * 4 + 127) / 128 * 128,
                       uv = dT + 4 * E2 * 12 * 4, rowbuf = uv + 128 * 20 * 4, total = rowbuf + kSplitRowCap * 16;
};

template <int E0, int E1, int E2>
__global__ void __launch_bounds__(kSplitThreads, 2) k_split_bwd(DevModel M, SysDesc D, int ba,
                                                               const float4 *__restrict__ posS,
                                                               const float *__restrict__ box,
                                                               const int32_t *__restrict__ nbrs,
                                                               const float4 *__restrict__ rows_g,
                                                               const int *__restrict__ rcnt,
                                                               const float *__restrict__ dT, ForceSum *__restrict__ F4,
                                                               double *__restrict__ virial, int *__restrict__ err) {
  using SD = SplitDims<E0, E1, E2>;
  using SM = SplitBwdSmem<E0, E1, E2>;
  extern __shared__ __align__(1024) char smem[];
  char *netb = smem + SM::net;
  float *sm = reinterpret_cast<float *>(smem + SM::small);
  float *dTs = reinterpret_cast<float *>(smem + SM::dT), *uvs = reinterpret_cast<float *>(smem + SM::uv);
  float4 *rowbuf = reinterpret_cast<float4 *>(smem + SM::rowbuf);
  __shared__ int wcnt[kSplitThreads / 32];
  __shared__ float3 ri_s[kBlkAtoms];
  __shared__ int src_s[4];  // user index of each centre
  __shared__ double vir_s[9];
  __shared__ float wvir_s[4][9];
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
  const uint32_t tX = tbase + kTmX, tY = tbase + kTmY;
  uint32_t ph = 0;
  bool ok = true;
  const uint32_t idesc1 = tc::idesc_f16(128, SD::N1, 0, 0), idesc2 = tc::idesc_f16(128, SD::NP, 0, 0);
  const uint32_t w1_u = tc::smem_u32(netb), w2_u = w1_u + 2 * SD::W1B;
  // the virial of the rows of one block in FP32, from block to block in FP64
  float vir[9];
#pragma unroll
  for (int k = 0; k < 9; ++k) vir[k] = 0.f;
  int vframe = -1;
  const int nblk = blocks_total(D, ba);
  int loaded_net = -1;

  for (int blk = blockIdx.x; blk < nblk && ok; blk += gridDim.x) {
    const BlkPos bp = block_pos(D, ba, blk);
    const int ti = bp.ti, nb = bp.nb, f = bp.f;
    const size_t g0 = bp.g0, frame_base = (size_t)f * D.N;
    const float inv_std = M.inv_std[ti], mean = M.mean[ti];
    if (blk + (int)gridDim.x < nblk) {
      const BlkPos bn = block_pos(D, ba, blk + gridDim.x);
      if (rows_g != nullptr && D.S <= kRowStoreCap)
        prefetch_range_l2(rows_g + bn.g0 * kRowStoreCap, (size_t)bn.nb * D.S * 16);
      else prefetch_range_l2(nbrs + bn.g0 * D.S, (size_t)bn.nb * D.S * 4);
      prefetch_range_l2(dT + bn.g0 * 10 * E2, (size_t)bn.nb * 10 * E2 * 4);
    }
    const int bs = box_slot(D, g0, f);
    if (bs != vframe && tid < 9) {
      if (vframe >= 0) {
        atomicAdd(&virial[vframe * 9 + tid], vir_s[tid]);
        vir_s[tid] = 0.0;
      }
    }
    vframe = bs;
    const float3 L = make_float3(box[bs * 3], box[bs * 3 + 1], box[bs * 3 + 2]);
    const int3 ni = image_range(L, M.rcut);
    const int nim = (2 * ni.x + 1) * (2 * ni.y + 1) * (2 * ni.z + 1);
    const bool stream = row_store_covers(D, rows_g, nim);
    if (tid < nb) {
      const float4 q = posS[g0 + tid];
      ri_s[tid] = make_float3(q.x, q.y, q.z);
      src_s[tid] = __float_as_int(q.w);
    }
    for (int e = tid; e < nb * 10 * E2; e += kSplitThreads) {  // dT rows [slot][c][w] -> [slot][w][12]
      const int sc = e / E2, w = e - sc * E2, slot = sc / 10, c = sc - slot * 10;
      dTs[(slot * E2 + w) * 12 + c] = dT[g0 * 10 * E2 + e];
    }
    __syncthreads();
    int rowstart = 0, rowcount = 0;
    const int tj0 = (loaded_net >= 0 && loaded_net / M.ntypes == ti) ? loaded_net - ti * M.ntypes : 0;
    for (int tt = 0; tt < D.ntypes && ok; ++tt) {
      const int tj = (tj0 + tt) % D.ntypes;
      const int per_atom = D.sel[tj] * nim, total = nb * per_atom;
      const int knet = ti * M.ntypes + tj;
      const float4 *rsrc = stream ? rows_g + g0 * kRowStoreCap + (size_t)nb * D.col[tj] : nullptr;
      const int nsrc = stream ? rcnt[g0 * M.ntypes + tj] : total;
      for (int base = 0; base < nsrc + kSplitThreads && ok; base += kSplitThreads) {
        const bool flush = base >= nsrc;
        if (!flush) {
          if (stream) mix_stream_round<1>(rsrc, base, nsrc, rowbuf, rowstart, rowcount);
          else
            mix_compact_round<1>(D, M, tj, base, total, per_atom, nim, ni, L, g0, frame_base, ri_s, posS, nbrs, rowbuf,
                                 wcnt, rowstart, rowcount);
        }
        while (rowcount - rowstart >= 128 || (flush && rowcount > rowstart)) {
          const int nrows = min(rowcount - rowstart, 128);
          if (loaded_net != knet) {
            __syncthreads();
            split_load_net<E0, E1, E2>(M, knet, netb, sm);
            loaded_net = knet;
          }
          const bool act = row < nrows;
          const float4 rv = act ? rowbuf[rowstart + row] : make_float4(100.f, 100.f, 100.f, 0.f);
          const int packed = act ? __float_as_int(rv.w) : 0;
          const int slot = packed & 7;
          float st;
          {
            RowGeom gm;
            row_geom(make_float3(rv.x, rv.y, rv.z), M.rcut, gm);
            st = (gm.s - mean) * inv_std;
          }
          tc::cp_async_wait<0>();
          __syncthreads();  // net image visible; rowbuf read; the previous tile's partial sums read
          f2 h1[SD::H1N / 2], d1[SD::H1N / 2];
          {
            f2 h0[SD::H0N / 2], d0[SD::H0N / 2];
            if (half == 0) split_layer0<E0, E1, E2, 0, true>(st, sm, tY + lane_off, h0, d0);
            else split_layer0<E0, E1, E2, 1, true>(st, sm, tY + lane_off, h0, d0);
            tc::tmem_wait_st();
            tc::fence_proxy_async();
            tc::fence_before_sync();
            __syncthreads();
            if (warp == 0 && tc::elect_one()) {
              tc::fence_after_sync();
              split_mma<SD::K1>(tX, tY, w1_u, SD::W1B, idesc1);
              split_mma<SD::K1>(tX + SD::N1, tY + SD::K1, w1_u, SD::W1B, idesc1);
              tc::commit(&mbar);
            }
            MIX_WAIT();
            if (!ok) break;
            if (half == 0) split_layer1<E0, E1, E2, 0, true>(tX + lane_off, tY + lane_off, sm, h0, d0, h1, d1);
            else split_layer1<E0, E1, E2, 1, true>(tX + lane_off, tY + lane_off, sm, h0, d0, h1, d1);
          }
          f2 u[5], v[5];
#pragma unroll
          for (int c = 0; c < 5; ++c) u[c] = v[c] = tc::pk1(0.f);
          const float *dTr = dTs + slot * E2 * 12;
#pragma unroll
          for (int pass = 0; pass < 2; ++pass) {
            tc::tmem_wait_st();
            tc::fence_before_sync();
            __syncthreads();  // A1 written (pass 0); the accumulators of pass 0 read (pass 1)
            if (warp == 0 && tc::elect_one()) {
              tc::fence_after_sync();
              const uint32_t wp = w2_u + pass * 2 * SD::W2B;
              split_mma<SD::K2>(tX, tY, wp, SD::W2B, idesc2);
              split_mma<SD::K2>(tX + SD::NP, tY + SD::K2, wp, SD::W2B, idesc2);
              tc::commit(&mbar);
            }
            MIX_WAIT();
            if (!ok) break;
            const f2 us = tc::pk1(sm[SD::O_SC + 1]), one = tc::pk1(1.f);
            auto epi2 = [&](auto HALF) {
              constexpr int H = decltype(HALF)::value, P = H ? SD::P1 : SD::P0;
#pragma unroll
              for (int g = 0; g < P; g += 8) {
                uint32_t z[8], dz[8];
                tc::tmem_ld8_issue(tX + lane_off + H * SD::HP + g, z);
                tc::tmem_ld8_issue(tX + lane_off + SD::NP + H * SD::HP + g, dz);
                tc::tmem_wait();
#pragma unroll
                for (int i = 0; i < 8; i += 2)
                  if (g + i < P) {
                    const int pc = pass * P + g + i;
                    const f2 b = *reinterpret_cast<const f2 *>(sm + SD::O_B2 + pass * SD::NP + H * SD::HP + g + i);
                    const f2 t =
                        tc::tanh_pair(tc::fma2(tc::pk(__uint_as_float(z[i]), __uint_as_float(z[i + 1])), us, b));
                    const f2 h2 = tc::add2(t, split_res<SD::Z2>(h1, pc));
                    const f2 g2 = tc::mul2(tc::fma2(tc::mul2(t, tc::pk1(-1.f)), t, one), us);
                    const f2 dh2 = tc::fma2(g2, tc::pk(__uint_as_float(dz[i]), __uint_as_float(dz[i + 1])),
                                            split_res<SD::Z2>(d1, pc));
                    float ha, hb, da, db;
                    tc::upk(h2, ha, hb);
                    tc::upk(dh2, da, db);
                    const float *q = dTr + (H * SD::S2 + pc) * 12;
#pragma unroll
                    for (int k = 0; k < 2; ++k, q += 12) {
                      const f2 hh = tc::pk1(k ? hb : ha), dd = tc::pk1(k ? db : da);
                      const float4 q0 = *reinterpret_cast<const float4 *>(q), q1 = *reinterpret_cast<const float4 *>(q + 4);
                      const float2 q2 = *reinterpret_cast<const float2 *>(q + 8);
                      const f2 w[5] = {tc::pk(q0.x, q0.y), tc::pk(q0.z, q0.w), tc::pk(q1.x, q1.y), tc::pk(q1.z, q1.w),
                                       tc::pk(q2.x, q2.y)};
#pragma unroll
                      for (int c = 0; c < 5; ++c) {
                        u[c] = tc::fma2(hh, w[c], u[c]);
                        v[c] = tc::fma2(dd, w[c], v[c]);
                      }
                    }
                  }
              }
            };
            if (half == 0) epi2(std::integral_constant<int, 0>());
            else epi2(std::integral_constant<int, 1>());
          }
          if (!ok) break;
          tc::fence_before_sync();
          f2 *ux = reinterpret_cast<f2 *>(uvs + row * 20);
          if (half == 1) {
#pragma unroll
            for (int c = 0; c < 5; ++c) {
              ux[c] = u[c];
              ux[5 + c] = v[c];
            }
          }
          __syncthreads();
          if (half == 0) {
            float uu[10], vv[10];
#pragma unroll
            for (int c = 0; c < 5; ++c) {
              tc::upk(tc::add2(u[c], ux[c]), uu[2 * c], uu[2 * c + 1]);
              tc::upk(tc::add2(v[c], ux[5 + c]), vv[2 * c], vv[2 * c + 1]);
            }
            RowGeom gm;
            float st2, R[10], gst = 0.f;
            split_row_env(rv, M.rcut, inv_std, mean, gm, st2, R);
#pragma unroll
            for (int c = 0; c < 10; ++c) gst = fmaf(R[c], vv[c], gst);
            float gx[3];
            row_adjoint(gm, inv_std, uu, gst * sm[SD::O_SC + 2], gx);
            if (act) {
              force_add(F4[frame_base + (packed >> 3)], -gx[0], -gx[1], -gx[2]);
#pragma unroll
              for (int p3 = 0; p3 < 3; ++p3)
#pragma unroll
                for (int q3 = 0; q3 < 3; ++q3) vir[p3 * 3 + q3] -= gm.x[p3] * gx[q3];
            }
            // centre force: rows are sorted by slot, a segmented suffix sum
            // leaves each slot's total on its first lane
            const int key = act ? slot : -1 - lane;
            float s0 = act ? gx[0] : 0.f, s1 = act ? gx[1] : 0.f, s2 = act ? gx[2] : 0.f;
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
    if (half == 0) {
#pragma unroll
      for (int k = 0; k < 9; ++k) {
        const float s = warp_sum(vir[k]);
        if (lane == 0) wvir_s[warp][k] = s;
        vir[k] = 0.f;
      }
    }
    __syncthreads();
    if (tid < 9)
      vir_s[tid] += ((double)wvir_s[0][tid] + (double)wvir_s[1][tid]) + ((double)wvir_s[2][tid] + (double)wvir_s[3][tid]);
    __syncthreads();
  }
  if (!ok) {
    if (tid == 0) atomicOr(err, 1);  // a tensor-core wait gave up (k_finalize)
    tc::mbar_wait(&mbar, ph);
  }
  tc::cp_async_wait<0>();
  tc::fence_before_sync();
  __syncthreads();
  if (tid < 9 && vframe >= 0) atomicAdd(&virial[vframe * 9 + tid], vir_s[tid]);
  if (warp == 0) tc::tmem_dealloc(tbase, 256);
}

// ---------------------------------------------------------------- launches
static int split_sms() {
  int dev = 0, nsm = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  return nsm;
}

// Centre atoms per block: 4 fill the 128-row tiles best (about 87 % at liquid
// density); fewer when that leaves SMs without a block.
int split_block_atoms(const SysDesc &D) {
  const int want = 2 * split_sms();
  for (int ba = 4; ba > 1; ba >>= 1)
    if (blocks_total(D, ba) >= want) return ba;
  return 1;
}

template <int E0, int E1, int E2>
static int launch_fwd(const DevModel &M, const SysDesc &D, int ba, const float4 *posS, const float *box,
                      const int32_t *nbrs, const float4 *rows, const int *rcnt, float *T, float *G, float *gmax, int *err,
                      cudaStream_t st) {
  const int nblk = blocks_total(D, ba), smem = SplitFwdSmem<E0, E1, E2>::total;
  if (!nblk) return DPB_OK;
  DPB_CUDA_TRY(cudaFuncSetAttribute(k_split_fwd<E0, E1, E2>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  const int grid = std::min(nblk, 2 * split_sms());
  k_split_fwd<E0, E1, E2><<<grid, kSplitThreads, smem, st>>>(M, D, ba, posS, box, nbrs, rows, rcnt, T, G, gmax, err);
  count_launch();
  DPB_LAUNCH_CHECK();
  return DPB_OK;
}

template <int E0, int E1, int E2>
static int launch_bwd(const DevModel &M, const SysDesc &D, int ba, const float4 *posS, const float *box,
                      const int32_t *nbrs, const float4 *rows, const int *rcnt, float *T, const float *dG, ForceSum *F4,
                      double *virial, int *err, cudaStream_t st) {
  const int nblk = blocks_total(D, ba), smem = SplitBwdSmem<E0, E1, E2>::total;
  if (!nblk) return DPB_OK;
  const size_t NF = (size_t)D.N * D.F;
  const int dsm = 4 * SplitDtSmem<E2>::floats * 4;
  DPB_CUDA_TRY(cudaFuncSetAttribute(k_split_dT<E2>, cudaFuncAttributeMaxDynamicSharedMemorySize, dsm));
  const unsigned dgrid = (unsigned)std::min((NF + 3) / 4, (size_t)split_sms() * kSplitDtCtas);
  k_split_dT<E2><<<dgrid, 128, dsm, st>>>(M, (int)NF, T, dG);
  count_launch();
  DPB_LAUNCH_CHECK();
  DPB_CUDA_TRY(cudaFuncSetAttribute(k_split_bwd<E0, E1, E2>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  const int grid = std::min(nblk, 2 * split_sms());
  k_split_bwd<E0, E1, E2><<<grid, kSplitThreads, smem, st>>>(M, D, ba, posS, box, nbrs, rows, rcnt, T, F4, virial, err);
  count_launch();
  DPB_LAUNCH_CHECK();
  return DPB_OK;
}

int split_embed_fwd(const DevModel &M, const SysDesc &D, int ba, const float4 *posS, const float *box,
                    const int32_t *nbrs, const float4 *rows, const int *rcnt, float *T, float *G, float *gmax, int *err,
                    cudaStream_t st) {
  return M.E2 == 100 ? launch_fwd<25, 50, 100>(M, D, ba, posS, box, nbrs, rows, rcnt, T, G, gmax, err, st)
                     : launch_fwd<32, 32, 64>(M, D, ba, posS, box, nbrs, rows, rcnt, T, G, gmax, err, st);
}

int split_embed_bwd(const DevModel &M, const SysDesc &D, int ba, const float4 *posS, const float *box,
                    const int32_t *nbrs, const float4 *rows, const int *rcnt, float *T, const float *dG, ForceSum *F4,
                    double *virial, int *err, cudaStream_t st) {
  return M.E2 == 100 ? launch_bwd<25, 50, 100>(M, D, ba, posS, box, nbrs, rows, rcnt, T, dG, F4, virial, err, st)
                     : launch_bwd<32, 32, 64>(M, D, ba, posS, box, nbrs, rows, rcnt, T, dG, F4, virial, err, st);
}

}  // namespace dpb

// FP32 evaluation with compressed embedding tables, and the pieces that every
// FP32 evaluation shares (reference model: deepmd_jax/dpmodel.py:30-100,
// embedding/fitting nets deepmd_jax/utils.py:100-166):
//   k_embed_fwd   warp per centre atom: neighbour rows with s(r) != 0 are
//                 compacted, looked up in the type pair's table, contracted with
//                 the 10-channel env rows into T (10 x W); the epilogue forms
//                 the descriptor G (A x W) and its largest entry.
//   k_embed_bwd   warp per centre atom: dE/dT from dE/dG, then the rows' h and
//                 dh/ds~ give dE/ds~ and dE/dR~; the row adjoint gives dE/dx,
//                 scattered as forces (FP64 atomics) and reduced into the
//                 virial.
//   k_fit_energy, k_finalize
// The tuned uncompressed nets run in embed_split.cu, other shapes in
// eval_general.cu, the fitting net in gemm_split.cu.
// Rows with s(r) = 0 contribute exactly zero in the reference (R~ = 0) and are
// skipped here.
#include "eval_common.cuh"

namespace dpb {

__device__ __forceinline__ float3 load_pos(const float *__restrict__ pos, const int32_t *__restrict__ perm,
                                           int f, int k, int N) {
  int src = perm ? perm[k] : k;
  const float *p = pos + ((size_t)f * N + src) * 3;
  return make_float3(p[0], p[1], p[2]);
}

// ---------------------------------------------------------------- compressed embedding
// The table lookup of the compressed embedding net (deepmd_jax/utils.py:126-151):
// x = s~ - srmin; idx = trunc(x / delta); x0 = x - idx * delta; the gather
// clamps idx into [0, Ngrids) while x0 keeps the unclamped idx; h[w] =
// sum_i c[idx][i][w] x0^(5-i), evaluated here by Horner's rule.
__device__ __forceinline__ void cmp_locate(float st, float srmin, float delta, int ng, int &idx, float &x0) {
  const float x = __fsub_rn(st, srmin);
  const int k = (int)__fdiv_rn(x, delta);  // truncation toward zero, like astype(int)
  x0 = __fsub_rn(x, __fmul_rn((float)k, delta));
  idx = k < 0 ? 0 : (k >= ng ? ng - 1 : k);
}

// One round of up to 32 compacted rows, column-parallel: a lane owns VC
// neighbouring columns, so that one pass over the rows covers all of them; the
// rows' (idx, x0) and env rows are read from the row buffer (st slot overwritten
// by x0, slot 11 by idx) as three 16-byte words and each table row is read with
// coalesced loads.  T += R~^T h accumulates into the warp's shared T.  (With one
// column per lane, two or four passes of twelve 4-byte reads per row: 206 us for
// 12,288 atoms of width 64, 170 us now.)
template <int E2>
__device__ __forceinline__ void embed_rows_fwd_cmp(const float *__restrict__ coeff, float srmin, float delta,
                                                   int ng, int n, float *__restrict__ rowbuf,
                                                   float *__restrict__ Ts, int lane) {
  constexpr int VC = E2 <= 64 ? 2 : 4;
  static_assert(E2 % VC == 0 && E2 / VC <= 32, "columns per lane");
  if (lane < n) {
    int idx;
    float x0;
    cmp_locate(rowbuf[lane * 12], srmin, delta, ng, idx, x0);
    rowbuf[lane * 12] = x0;
    rowbuf[lane * 12 + 11] = __int_as_float(idx);
  }
  __syncwarp();
  if (lane < E2 / VC) {
    const int col = VC * lane;
    float Tq[10][VC];
#pragma unroll
    for (int c = 0; c < 10; ++c)
#pragma unroll
      for (int e = 0; e < VC; ++e) Tq[c][e] = 0.f;
#pragma unroll 2
    for (int r = 0; r < n; ++r) {
      const float4 *rb = reinterpret_cast<const float4 *>(rowbuf + r * 12);
      const float4 w0 = rb[0], w1 = rb[1], w2 = rb[2];
      const float R[10] = {w0.y, w0.z, w0.w, w1.x, w1.y, w1.z, w1.w, w2.x, w2.y, w2.z};
      const float x0 = w0.x;
      const float *cr = coeff + (size_t)__float_as_int(w2.w) * 6 * E2 + col;
      float cf[6][VC];
#pragma unroll
      for (int i = 0; i < 6; ++i) {
        if constexpr (VC == 2) {
          const float2 t = __ldg(reinterpret_cast<const float2 *>(cr + i * E2));
          cf[i][0] = t.x; cf[i][1] = t.y;
        } else {
          const float4 t = __ldg(reinterpret_cast<const float4 *>(cr + i * E2));
          cf[i][0] = t.x; cf[i][1] = t.y; cf[i][2] = t.z; cf[i][3] = t.w;
        }
      }
#pragma unroll
      for (int e = 0; e < VC; ++e) {
        float h = cf[0][e];
#pragma unroll
        for (int i = 1; i < 6; ++i) h = fmaf(h, x0, cf[i][e]);
#pragma unroll
        for (int c = 0; c < 10; ++c) Tq[c][e] = fmaf(R[c], h, Tq[c][e]);
      }
    }
#pragma unroll
    for (int c = 0; c < 10; ++c)
#pragma unroll
      for (int e = 0; e < VC; ++e) Ts[c * E2 + col + e] += Tq[c][e];
  }
  __syncwarp();
}

template <int E2>
__host__ __device__ constexpr int embed_fwd_warp_floats() {
  return 64 * 12 + 10 * E2;
}

template <int E2>
__global__ void __launch_bounds__(256) k_embed_fwd(DevModel M, SysDesc D, int ti, const float *__restrict__ pos,
                                                   const int32_t *__restrict__ perm, const float *__restrict__ box,
                                                   const int32_t *__restrict__ nbrs, float *__restrict__ Tout,
                                                   float *__restrict__ Gout, float *__restrict__ gmax) {
  extern __shared__ __align__(16) float smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, wpb = blockDim.x >> 5;
  float *rowbuf = smem + warp * embed_fwd_warp_floats<E2>();
  float *Ts = rowbuf + 64 * 12;
  const int f = blockIdx.y;
  const int a = blockIdx.x * wpb + warp;
  const int cnt_i = D.offs[ti + 1] - D.offs[ti];
  if (a >= cnt_i) return;
  const int i = D.offs[ti] + a;
  const size_t g = (size_t)f * D.N + i;
  const float3 ri = load_pos(pos, perm, f, i, D.N);
  const int bs = box_slot(D, g, f);
  const float3 L = make_float3(box[bs * 3], box[bs * 3 + 1], box[bs * 3 + 2]);
  const int3 ni = image_range(L, M.rcut);
  const int nim = (2 * ni.x + 1) * (2 * ni.y + 1) * (2 * ni.z + 1);
  const float inv_std = M.inv_std[ti], mean = M.mean[ti];
  const unsigned lt = (1u << lane) - 1u;
  for (int e = lane; e < 10 * E2; e += 32) Ts[e] = 0.f;
  __syncwarp();

  for (int tj = 0; tj < D.ntypes; ++tj) {
    const int32_t *nb = nbrs + g * D.S + D.col[tj];
    const int sel = D.sel[tj], cnt_j = D.offs[tj + 1] - D.offs[tj];
    int nbuf = 0;
    const int total = sel * nim;
    for (int base = 0; base < total; base += 32) {
      const int p = base + lane;
      bool keep = false;
      float st = 0.f, R[10];
      if (p < total) {
        const int slot = nim == 1 ? p : p / nim, mimg = p - slot * nim;
        const int idx = nb[slot] & DPB_NBR_INDEX_MASK;
        if (idx < cnt_j) {
          const float3 rj = load_pos(pos, perm, f, D.offs[tj] + idx, D.N);
          RowGeom gm;
          row_geom(rel_coord(ri, rj, L, ni, mimg), M.rcut, gm);
          if (gm.s != 0.f) {
            keep = true;
            const float sn = gm.s * inv_std;
            st = (gm.s - mean) * inv_std;
            const float inv_rp = 1.f / (gm.r + 1e-16f);
            const float xh[3] = {gm.x[0] * inv_rp, gm.x[1] * inv_rp, gm.x[2] * inv_rp};
            env_row(sn, xh, R);
          }
        }
      }
      const unsigned m = __ballot_sync(0xffffffffu, keep);
      if (keep) {
        float *dst = rowbuf + (nbuf + __popc(m & lt)) * 12;
        dst[0] = st;
#pragma unroll
        for (int c = 0; c < 10; ++c) dst[1 + c] = R[c];
      }
      nbuf += __popc(m);
      __syncwarp();
      if (nbuf >= 32) {
        embed_rows_fwd_cmp<E2>(M.cmp_coeff[ti * M.ntypes + tj], M.cmp_srmin[ti * M.ntypes + tj],
                               M.cmp_delta[ti * M.ntypes + tj], M.ngrids, 32, rowbuf, Ts, lane);
        const int rem = nbuf - 32;
        if (lane < rem)
          for (int c = 0; c < 12; ++c) rowbuf[lane * 12 + c] = rowbuf[(32 + lane) * 12 + c];
        __syncwarp();
        nbuf = rem;
      }
    }
    if (nbuf > 0) {
      embed_rows_fwd_cmp<E2>(M.cmp_coeff[ti * M.ntypes + tj], M.cmp_srmin[ti * M.ntypes + tj],
                             M.cmp_delta[ti * M.ntypes + tj], M.ngrids, nbuf, rowbuf, Ts, lane);
    }
    __syncwarp();
  }

  // T = sum / Nnbrs (written out); Ts becomes X = T with Tbias on channel 0
  for (int e = lane; e < 10 * E2; e += 32) {
    const float t = Ts[e] * M.inv_nnbrs;
    Tout[g * 10 * E2 + e] = t;
    Ts[e] = t + (e < E2 ? M.tbias[e] : 0.f);
  }
  __syncwarp();
  // G[a][w] = sum_c Q[c][a] X[c][w] (dpmodel.py:74-78), Q[c<4][a] = X[c][a],
  // Q[4+m][a] = tensor_3to6(X[1:4][A+a])[m] + X[4+m][A+a]
  const int A = M.A;
  float *Gg = Gout + g * (size_t)A * E2;
  float gm = 0.f;
  for (int aa = 0; aa < A; ++aa) {
    float Q[10];
#pragma unroll
    for (int c = 0; c < 4; ++c) Q[c] = Ts[c * E2 + aa];
    const float y1 = Ts[1 * E2 + A + aa], y2 = Ts[2 * E2 + A + aa], y3 = Ts[3 * E2 + A + aa];
    Q[4] = y1 * y1 + Ts[4 * E2 + A + aa];
    Q[5] = y2 * y2 + Ts[5 * E2 + A + aa];
    Q[6] = y3 * y3 + Ts[6 * E2 + A + aa];
    Q[7] = kSqrt2 * y1 * y3 + Ts[7 * E2 + A + aa];
    Q[8] = kSqrt2 * y2 * y1 + Ts[8 * E2 + A + aa];
    Q[9] = kSqrt2 * y3 * y2 + Ts[9 * E2 + A + aa];
    for (int col = lane; col < E2; col += 32) {
      float v = 0.f;
#pragma unroll
      for (int c = 0; c < 10; ++c) v = fmaf(Q[c], Ts[c * E2 + col], v);
      Gg[aa * E2 + col] = v;
      gm = fmaxf(gm, fabsf(v));
    }
  }
  if (gmax) {  // the fitting GEMM's row scale
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) gm = fmaxf(gm, __shfl_xor_sync(0xffffffffu, gm, o));
    if (lane == 0) gmax[g] = gm;
  }
}

// ---------------------------------------------------------------- adjoint
// Adjoint of one round of rows of a compressed net: h and dh/ds~ = dh/dx0 from
// the rows' table entries, u = dT.h, v = dT.dh, then (row = lane) the same
// env-row adjoint as the MLP path.  The table entries of 16 rows are read 32
// columns at a time, 8 lanes on one row's whole line, and h and dh go through
// shared memory to two lanes per row for the sums.  (With row = lane every load
// touched 32 lines at the same offset: up to 32 tag lookups and 8-way conflicts
// per instruction, 3,000 clocks per round of 32 rows: 637 us for 12,288 atoms of
// width 64, 413 us now.)
constexpr int kCmpS = 36;                    // row stride of h and dh (floats)
constexpr int kCmpHd = 2 * 16 * kCmpS;       // floats of both
template <int E2>
__device__ __forceinline__ void embed_rows_bwd_cmp(const float *__restrict__ coeff, float srmin, float delta,
                                                   int ng, int n, const float *__restrict__ rowbuf,
                                                   float *__restrict__ hd, const float *__restrict__ dT,
                                                   float inv_std, float mean, int lane, float &fi0, float &fi1,
                                                   float &fi2, float (&vir)[9], ForceSum *__restrict__ F4,
                                                   size_t frame_base) {
  static_assert(E2 % 4 == 0, "table width");
  const bool act = lane < n;
  RowGeom gm;
  int jj = 0;
  if (act) {
    const float *rb = rowbuf + lane * 8;
    gm.x[0] = rb[0]; gm.x[1] = rb[1]; gm.x[2] = rb[2];
    gm.r = rb[3]; gm.s = rb[4]; gm.dsdr = rb[5];
    jj = __float_as_int(rb[6]);
  } else {
    gm.x[0] = gm.x[1] = gm.x[2] = 0.f; gm.r = 1.f; gm.s = 0.f; gm.dsdr = 0.f;
  }
  const float sn = gm.s * inv_std, st = (gm.s - mean) * inv_std;
  int idx;
  float x0;
  cmp_locate(st, srmin, delta, ng, idx, x0);
  float u[10], v[10];
  const int half = lane >> 4, cq = 4 * (lane & 7);
#pragma unroll 1
  for (int b = 0; 16 * b < n; ++b) {  // rows 16 b .. 16 b + 15
    float us[10], vs[10];
#pragma unroll
    for (int c = 0; c < 10; ++c) us[c] = vs[c] = 0.f;
#pragma unroll 1
    for (int c0 = 0; c0 < E2; c0 += 32) {
      __syncwarp();
#pragma unroll 2
      for (int p = 0; p < 4; ++p) {
        const int r = 4 * p + (lane >> 3);
        const int id = __shfl_sync(0xffffffffu, idx, 16 * b + r);
        const float x = __shfl_sync(0xffffffffu, x0, 16 * b + r);
        if (E2 % 32 == 0 || c0 + cq < E2) {
          const float4 *cr = reinterpret_cast<const float4 *>(coeff + (size_t)id * 6 * E2 + c0 + cq);
          float4 c[6];
#pragma unroll
          for (int i = 0; i < 6; ++i) c[i] = __ldg(cr + i * (E2 / 4));
          const float cc[6][4] = {{c[0].x, c[0].y, c[0].z, c[0].w}, {c[1].x, c[1].y, c[1].z, c[1].w},
                                  {c[2].x, c[2].y, c[2].z, c[2].w}, {c[3].x, c[3].y, c[3].z, c[3].w},
                                  {c[4].x, c[4].y, c[4].z, c[4].w}, {c[5].x, c[5].y, c[5].z, c[5].w}};
          float h[4], dh[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            h[e] = cc[0][e];
            dh[e] = 5.f * cc[0][e];
#pragma unroll
            for (int i = 1; i < 5; ++i) {
              h[e] = fmaf(h[e], x, cc[i][e]);
              dh[e] = fmaf(dh[e], x, (float)(5 - i) * cc[i][e]);
            }
            h[e] = fmaf(h[e], x, cc[5][e]);
          }
          *reinterpret_cast<float4 *>(hd + r * kCmpS + cq) = make_float4(h[0], h[1], h[2], h[3]);
          *reinterpret_cast<float4 *>(hd + kCmpHd / 2 + r * kCmpS + cq) = make_float4(dh[0], dh[1], dh[2], dh[3]);
        }
      }
      __syncwarp();
#pragma unroll 2
      for (int q = 0; q < 4; ++q) {
        const int k = 16 * half + 4 * q, col = c0 + k;
        if (E2 % 32 == 0 || col < E2) {
          const float4 h = *reinterpret_cast<const float4 *>(hd + (lane & 15) * kCmpS + k);
          const float4 d = *reinterpret_cast<const float4 *>(hd + kCmpHd / 2 + (lane & 15) * kCmpS + k);
#pragma unroll
          for (int ch = 0; ch < 10; ++ch) {
            const float4 t = *reinterpret_cast<const float4 *>(dT + ch * (E2 + 4) + col);
            us[ch] = fmaf(t.w, h.w, fmaf(t.z, h.z, fmaf(t.y, h.y, fmaf(t.x, h.x, us[ch]))));
            vs[ch] = fmaf(t.w, d.w, fmaf(t.z, d.z, fmaf(t.y, d.y, fmaf(t.x, d.x, vs[ch]))));
          }
        }
      }
    }
#pragma unroll
    for (int c = 0; c < 10; ++c) {  // the two lanes of a row
      const float uc = us[c] + __shfl_xor_sync(0xffffffffu, us[c], 16);
      const float vc = vs[c] + __shfl_xor_sync(0xffffffffu, vs[c], 16);
      if (b == 0 || half == b) {
        u[c] = uc;
        v[c] = vc;
      }
    }
  }
  __syncwarp();
  const float inv_rp = 1.f / (gm.r + 1e-16f);
  const float xh[3] = {gm.x[0] * inv_rp, gm.x[1] * inv_rp, gm.x[2] * inv_rp};
  float R[10];
  env_row(sn, xh, R);
  float gst = 0.f;
#pragma unroll
  for (int c = 0; c < 10; ++c) gst = fmaf(R[c], v[c], gst);
  float gx[3];
  row_adjoint(gm, inv_std, u, gst, gx);
  if (act) {
    force_add(F4[frame_base + jj], -gx[0], -gx[1], -gx[2]);
    fi0 += gx[0]; fi1 += gx[1]; fi2 += gx[2];
#pragma unroll
    for (int p = 0; p < 3; ++p)
#pragma unroll
      for (int qq = 0; qq < 3; ++qq) vir[p * 3 + qq] -= gm.x[p] * gx[qq];
  }
}

// Floats of a warp's dG (row stride E2 + 1), later its 64 rows and h and dh.
template <int E2>
__host__ __device__ __forceinline__ int cmp_bwd_r1(int A) {
  const int a = (A * (E2 + 1) + 3) / 4 * 4, b = 64 * 8 + kCmpHd;
  return a > b ? a : b;
}

template <int E2>
__global__ void __launch_bounds__(256, 2) k_embed_bwd(DevModel M, SysDesc D, int ti, const float *__restrict__ pos,
                                                   const int32_t *__restrict__ perm, const float *__restrict__ box,
                                                   const int32_t *__restrict__ nbrs, const float *__restrict__ Tin,
                                                   const float *__restrict__ dG, ForceSum *__restrict__ F4,
                                                   double *__restrict__ virial) {
  constexpr int NQ = (E2 + 31) / 32;
  extern __shared__ __align__(16) float smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, wpb = blockDim.x >> 5;
  const int A = M.A;
  constexpr int AS = E2 + 1, BS = E2 + 4;  // row strides: dot products along rows without bank conflicts
  const int r1 = cmp_bwd_r1<E2>(A);
  const int per_warp = r1 + 10 * BS + 20 * A;
  float *bufA = smem + warp * per_warp;  // dG, later rows, h and dh
  float *bufB = bufA + r1;                                   // X, later dT
  float *Qs = bufB + 10 * BS;                                // 10 x A
  float *dQs = Qs + 10 * A;                                  // 10 x A
  __shared__ double vsm[9];
  if (threadIdx.x < 9) vsm[threadIdx.x] = 0.0;
  __syncthreads();
  const int f = blockIdx.y;
  const int a = blockIdx.x * wpb + warp;
  const int cnt_i = D.offs[ti + 1] - D.offs[ti];
  float vir[9];
#pragma unroll
  for (int k = 0; k < 9; ++k) vir[k] = 0.f;
  if (a < cnt_i) {
    const int i = D.offs[ti] + a;
    const size_t g = (size_t)f * D.N + i;
    // ---- dE/dT from dE/dG (adjoint of dpmodel.py:74-78)
    for (int e = lane; e < 10 * E2; e += 32) {
      const int c = e / E2, w = e - c * E2;
      bufB[c * BS + w] = Tin[g * 10 * E2 + e] + (c == 0 ? M.tbias[w] : 0.f);
    }
    for (int e = lane; e < A * E2; e += 32) bufA[e / E2 * AS + e % E2] = dG[g * (size_t)A * E2 + e];
    __syncwarp();
    for (int e = lane; e < 10 * A; e += 32) {
      const int c = e / A, aa = e - c * A;
      float qv;
      if (c < 4) {
        qv = bufB[c * BS + aa];
      } else {
        const float y1 = bufB[1 * BS + A + aa], y2 = bufB[2 * BS + A + aa], y3 = bufB[3 * BS + A + aa];
        const int m = c - 4;
        const float base[6] = {y1 * y1, y2 * y2, y3 * y3, kSqrt2 * y1 * y3, kSqrt2 * y2 * y1, kSqrt2 * y3 * y2};
        qv = base[m] + bufB[c * BS + A + aa];
      }
      Qs[e] = qv;
      float dq = 0.f;
      for (int w = 0; w < E2; ++w) dq = fmaf(bufA[aa * AS + w], bufB[c * BS + w], dq);
      dQs[e] = dq;
    }
    __syncwarp();
    float dX[NQ][10];
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
      const int col = q * 32 + lane;
#pragma unroll
      for (int c = 0; c < 10; ++c) dX[q][c] = 0.f;
      if (col < E2) {
        for (int aa = 0; aa < A; ++aa) {
          const float dg = bufA[aa * AS + col];
#pragma unroll
          for (int c = 0; c < 10; ++c) dX[q][c] = fmaf(dg, Qs[c * A + aa], dX[q][c]);
        }
      }
    }
    // row contributions through Q: channels 0..3 at w = a, G2 terms at w = A + a
    if (lane < A) {
#pragma unroll
      for (int c = 0; c < 4; ++c) dX[0][c] += dQs[c * A + lane];
    } else if (lane < 2 * A) {
      const int aa = lane - A;
      float d2[6];
#pragma unroll
      for (int m = 0; m < 6; ++m) d2[m] = dQs[(4 + m) * A + aa];
      const float y1 = bufB[1 * BS + lane], y2 = bufB[2 * BS + lane], y3 = bufB[3 * BS + lane];
#pragma unroll
      for (int m = 0; m < 6; ++m) dX[0][4 + m] += d2[m];
      dX[0][1] += 2.f * y1 * d2[0] + kSqrt2 * y3 * d2[3] + kSqrt2 * y2 * d2[4];
      dX[0][2] += 2.f * y2 * d2[1] + kSqrt2 * y1 * d2[4] + kSqrt2 * y3 * d2[5];
      dX[0][3] += 2.f * y3 * d2[2] + kSqrt2 * y1 * d2[3] + kSqrt2 * y2 * d2[5];
    }
    __syncwarp();
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
      const int col = q * 32 + lane;
      if (col < E2)
#pragma unroll
        for (int c = 0; c < 10; ++c) bufB[c * BS + col] = dX[q][c] * M.inv_nnbrs;
    }
    __syncwarp();
    // ---- rows: recompute with tangents, scatter forces
    const float3 ri = load_pos(pos, perm, f, i, D.N);
    const int bs = box_slot(D, g, f);
    const float3 L = make_float3(box[bs * 3], box[bs * 3 + 1], box[bs * 3 + 2]);
    const int3 ni = image_range(L, M.rcut);
    const int nim = (2 * ni.x + 1) * (2 * ni.y + 1) * (2 * ni.z + 1);
    const float inv_std = M.inv_std[ti], mean = M.mean[ti];
    const unsigned lt = (1u << lane) - 1u;
    float *rowbuf = bufA;  // 64 rows x 8 floats
    float fi0 = 0.f, fi1 = 0.f, fi2 = 0.f;
    const size_t frame_base = (size_t)f * D.N;
    for (int tj = 0; tj < D.ntypes; ++tj) {
        const int32_t *nb = nbrs + g * D.S + D.col[tj];
      const int sel = D.sel[tj], cnt_j = D.offs[tj + 1] - D.offs[tj];
      int nbuf = 0;
      const int total = sel * nim;
      for (int base = 0; base < total; base += 32) {
        const int p = base + lane;
        bool keep = false;
        RowGeom gm;
        int jj = 0;
        if (p < total) {
          const int slot = nim == 1 ? p : p / nim, mimg = p - slot * nim;
          const int idx = nb[slot] & DPB_NBR_INDEX_MASK;
          if (idx < cnt_j) {
            jj = D.offs[tj] + idx;
            const float3 rj = load_pos(pos, perm, f, jj, D.N);
            row_geom(rel_coord(ri, rj, L, ni, mimg), M.rcut, gm);
            keep = gm.s != 0.f;
          }
        }
        const unsigned m = __ballot_sync(0xffffffffu, keep);
        if (keep) {
          float *dst = rowbuf + (nbuf + __popc(m & lt)) * 8;
          dst[0] = gm.x[0]; dst[1] = gm.x[1]; dst[2] = gm.x[2];
          dst[3] = gm.r; dst[4] = gm.s; dst[5] = gm.dsdr;
          dst[6] = __int_as_float(perm ? perm[jj] : jj);
        }
        nbuf += __popc(m);
        __syncwarp();
        if (nbuf >= 32) {
          embed_rows_bwd_cmp<E2>(M.cmp_coeff[ti * M.ntypes + tj], M.cmp_srmin[ti * M.ntypes + tj],
                                 M.cmp_delta[ti * M.ntypes + tj], M.ngrids, 32, rowbuf, bufA + 64 * 8, bufB, inv_std, mean,
                                 lane, fi0, fi1, fi2, vir, F4, frame_base);
          const int rem = nbuf - 32;
          if (lane < rem)
            for (int c = 0; c < 8; ++c) rowbuf[lane * 8 + c] = rowbuf[(32 + lane) * 8 + c];
          __syncwarp();
          nbuf = rem;
        }
      }
      if (nbuf > 0) {
        embed_rows_bwd_cmp<E2>(M.cmp_coeff[ti * M.ntypes + tj], M.cmp_srmin[ti * M.ntypes + tj],
                               M.cmp_delta[ti * M.ntypes + tj], M.ngrids, nbuf, rowbuf, bufA + 64 * 8, bufB, inv_std, mean,
                               lane, fi0, fi1, fi2, vir, F4, frame_base);
      }
      __syncwarp();
    }
    fi0 = warp_sum(fi0); fi1 = warp_sum(fi1); fi2 = warp_sum(fi2);
    if (lane == 0) force_add(F4[frame_base + (perm ? perm[i] : i)], fi0, fi1, fi2);
  }
#pragma unroll
  for (int k = 0; k < 9; ++k) {
    float s = warp_sum(vir[k]);
    if (lane == 0 && s != 0.f) atomicAdd(&vsm[k], (double)s);
  }
  __syncthreads();
  // the block's 8 atoms share one frame (segment-aligned in packed batches)
  if (threadIdx.x < 9) {
    const int vs = box_slot(D, (size_t)f * D.N + D.offs[ti] + blockIdx.x * wpb, f);
    atomicAdd(&virial[vs * 9 + threadIdx.x], vsm[threadIdx.x]);
  }
}

// ---------------------------------------------------------------- fitting energy
// Per-atom energy E = H . w + b' and the first adjoint gate of the last hidden
// layer, gZ = w dt (1 - t^2): a warp per atom, 8 atoms per block (64 atoms per
// block with 8 in turn per warp took 27 us at 192 atoms, all latency); energies
// reduced in FP64, one atomic per run of one energy row.
__global__ void __launch_bounds__(256) k_fit_energy(EnergyArgs g, const float *__restrict__ H,
                                                    const float *__restrict__ tl, float *__restrict__ Eatom,
                                                    __half *__restrict__ gZ, int8_t *__restrict__ gexp,
                                                    double *__restrict__ energy, const int32_t *__restrict__ seg) {
  __shared__ double es[8];
  __shared__ int fs[8];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int ti = 0;
#pragma unroll
  for (int t = 1; t < kMaxTypes; ++t)
    if (t < g.ntypes && (int)blockIdx.x >= g.b0[t]) ti = t;
  const EnergyType &et = g.t[ti];
  const int r = ((int)blockIdx.x - g.b0[ti]) * 8 + warp;
  if (r < et.Mrows) {
    const size_t at = et.rm.atom(r);
    float s = 0.f;
    const int nc = (g.FWl + kGemmK - 1) / kGemmK, mt = g.mt0[ti] + r / 128, lr = r & 127;
    const float *h_ = H + at * g.FWl, *t_ = tl + at * g.FWl;
    const int n16 = (g.FWl + 15) / 16 * 16;  // whole K = 16 steps
    for (int n = 4 * lane; n - 4 * lane < n16; n += 128) {
      __align__(16) float h[4] = {0.f, 0.f, 0.f, 0.f}, t[4] = {1.f, 1.f, 1.f, 1.f}, w[4] = {0.f, 0.f, 0.f, 0.f};
      if ((g.FWl & 3) == 0 && n < g.FWl) {
        *reinterpret_cast<float4 *>(h) = *reinterpret_cast<const float4 *>(h_ + n);
        *reinterpret_cast<float4 *>(t) = *reinterpret_cast<const float4 *>(t_ + n);
      }
      float gz[4] = {0.f, 0.f, 0.f, 0.f}, gm = 0.f;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        if (n + e < g.FWl) {
          if ((g.FWl & 3) != 0) {
            h[e] = h_[n + e];
            t[e] = t_[n + e];
          }
          w[e] = et.wfin[n + e];
          s = fmaf(h[e], w[e], s);
          gz[e] = w[e] * (et.dtl ? et.dtl[n + e] : 1.f) * (1.f - t[e] * t[e]);
          gm = fmaxf(gm, fabsf(gz[e]));
        }
      }
#pragma unroll
      for (int o = 1; o < 8; o <<= 1) gm = fmaxf(gm, __shfl_xor_sync(0xffffffffu, gm, o));
      if (n >= n16) continue;
      const int k = gate_exp(gm);
      const float sc = pow2i(k);
      if ((lane & 7) == 0) gexp[gemm_exp_at(nc, mt, lr, n / kGemmK)] = (int8_t)k;
      __align__(8) __half hi[4], lo[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        hi[e] = __float2half_rn(gz[e] * sc);
        lo[e] = __float2half_rn(gz[e] * sc - __half2float(hi[e]));
      }
      __half *o = gZ + gemm_operand_at(nc, mt, lr, n);
      *reinterpret_cast<uint2 *>(o) = *reinterpret_cast<const uint2 *>(hi);
      *reinterpret_cast<uint2 *>(o + kGemmPart) = *reinterpret_cast<const uint2 *>(lo);
    }
    s = warp_sum(s) + et.bfin[0];
    if (lane == 0) {
      Eatom[at] = s;
      es[warp] = (double)s;
      fs[warp] = energy_slot(seg, at, g.N);
    }
  } else if (lane == 0) {
    es[warp] = 0.0;
    fs[warp] = -1;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double run = 0.0;
    int cf = fs[0];
    for (int k = 0; k < 8; ++k) {
      if (fs[k] != cf) {
        if (cf >= 0) atomicAdd(&energy[cf], run);
        run = 0.0;
        cf = fs[k];
      }
      run += es[k];
    }
    if (cf >= 0) atomicAdd(&energy[cf], run);
  }
}

// Forces (from their FP64 sums) and per-atom energies to the caller's layout;
// non-finite positions or results raise status bit 16 and, as NaN inputs do
// in the reference's float arithmetic, make the frame's energy NaN.  *err != 0:
// a tensor-core wait gave up, and what its CTA did not write is left from an
// earlier call, so every result is NaN.
__global__ void k_finalize(int NF, int N, const ForceSum *__restrict__ F4, float *__restrict__ force,
                           const float *__restrict__ Eatom_sorted, const int32_t *__restrict__ perm,
                           float *__restrict__ atom_energy, double *__restrict__ energy, int nE,
                           const float *__restrict__ pos, const int32_t *__restrict__ seg,
                           const int *__restrict__ err, uint32_t *__restrict__ status) {
  const int g = blockIdx.x * blockDim.x + threadIdx.x;
  const bool gave_up = err && *err != 0;
  const float nan = __int_as_float(0x7fffffff);
  if (g < NF) {
    const ForceSum a = F4[g];
    const float3 v = gave_up ? make_float3(nan, nan, nan) : make_float3((float)a.x, (float)a.y, (float)a.z);
    force[(size_t)g * 3 + 0] = v.x;
    force[(size_t)g * 3 + 1] = v.y;
    force[(size_t)g * 3 + 2] = v.z;
    const int f = g / N, k = g - f * N;
    const int dst = perm ? perm[k] : k;
    if (atom_energy) atom_energy[(size_t)f * N + dst] = gave_up ? nan : Eatom_sorted[g];
    const float *p = pos + ((size_t)f * N + dst) * 3;  // position of sorted atom g
    const bool bad_in = !isfinite(p[0]) || !isfinite(p[1]) || !isfinite(p[2]);
    if (bad_in || !isfinite(v.x) || !isfinite(v.y) || !isfinite(v.z)) atomicOr(status, DPB_ST_NONFINITE);
    const int e = energy_slot(seg, g, N);
    if (bad_in && e >= 0) energy[e] = __longlong_as_double(0x7ff8000000000000LL);
  }
  if (g < nE) {
    if (gave_up) energy[g] = __longlong_as_double(0x7ff8000000000000LL);
    if (gave_up || !isfinite(energy[g])) atomicOr(status, DPB_ST_NONFINITE);
  }
}

template <int E2>
int launch_embed_fwd_cmp(const DevModel &M, const SysDesc &D, int ti, const float *pos, const int32_t *perm,
                         const float *box, const int32_t *nbrs, float *T, float *G, float *gmax, cudaStream_t st) {
  const int cnt = D.offs[ti + 1] - D.offs[ti];
  if (cnt == 0) return DPB_OK;
  dim3 grid((cnt + 7) / 8, D.F);
  const size_t smem = (size_t)8 * embed_fwd_warp_floats<E2>() * sizeof(float);
  cudaFuncSetAttribute(k_embed_fwd<E2>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  k_embed_fwd<E2><<<grid, 256, smem, st>>>(M, D, ti, pos, perm, box, nbrs, T, G, gmax);
  count_launch();
  DPB_LAUNCH_CHECK();
  return DPB_OK;
}

template <int E2>
int launch_embed_bwd_cmp(const DevModel &M, const SysDesc &D, int ti, const float *pos, const int32_t *perm,
                         const float *box, const int32_t *nbrs, const float *T, const float *dG, ForceSum *F4,
                         double *virial, cudaStream_t st) {
  const int cnt = D.offs[ti + 1] - D.offs[ti];
  if (cnt == 0) return DPB_OK;
  dim3 grid((cnt + 7) / 8, D.F);
  const size_t smem = (size_t)8 * (cmp_bwd_r1<E2>(M.A) + 10 * (E2 + 4) + 20 * M.A) * sizeof(float);
  cudaFuncSetAttribute(k_embed_bwd<E2>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  k_embed_bwd<E2><<<grid, 256, smem, st>>>(M, D, ti, pos, perm, box, nbrs, T, dG, F4, virial);
  count_launch();
  DPB_LAUNCH_CHECK();
  return DPB_OK;
}

template int launch_embed_fwd_cmp<100>(const DevModel &, const SysDesc &, int, const float *, const int32_t *,
                                       const float *, const int32_t *, float *, float *, float *, cudaStream_t);
template int launch_embed_fwd_cmp<64>(const DevModel &, const SysDesc &, int, const float *, const int32_t *,
                                      const float *, const int32_t *, float *, float *, float *, cudaStream_t);
template int launch_embed_bwd_cmp<100>(const DevModel &, const SysDesc &, int, const float *, const int32_t *,
                                       const float *, const int32_t *, const float *, const float *, ForceSum *,
                                       double *, cudaStream_t);
template int launch_embed_bwd_cmp<64>(const DevModel &, const SysDesc &, int, const float *, const int32_t *,
                                      const float *, const int32_t *, const float *, const float *, ForceSum *, double *,
                                      cudaStream_t);

int launch_fit_energy(const EnergyArgs &g, const float *H, const float *tl, float *Eatom, __half *gZ, int8_t *gexp,
                      double *energy, const int32_t *seg, cudaStream_t st) {
  const int nb = g.b0[g.ntypes];
  if (nb == 0) return DPB_OK;
  k_fit_energy<<<nb, 256, 0, st>>>(g, H, tl, Eatom, gZ, gexp, energy, seg);
  count_launch();
  DPB_LAUNCH_CHECK();
  return DPB_OK;
}

int launch_finalize(int NF, int N, const ForceSum *F4, float *force, const float *Eatom, const int32_t *perm,
                    float *atom_energy, double *energy, int nE, const float *pos, const int32_t *seg,
                    const int *err, uint32_t *status, cudaStream_t st) {
  int n = NF > nE ? NF : nE;
  k_finalize<<<(n + 255) / 256, 256, 0, st>>>(NF, N, F4, force, Eatom, perm, atom_energy, energy, nE, pos, seg,
                                              err, status);
  count_launch();
  DPB_LAUNCH_CHECK();
  return DPB_OK;
}

}  // namespace dpb

extern "C" int dpb_selftest_finalize(int natoms, int nframes, const double *acc, const float *pos, const int *err,
                                     double *energy, float *atom_energy, float *force, uint32_t *status,
                                     void *stream) {
  if (natoms <= 0 || nframes <= 0 || !acc || !pos || !energy || !atom_energy || !force || !status ||
      (reinterpret_cast<uintptr_t>(acc) & 15) != 0)
    return DPB_ERR_INVALID_ARG;
  return dpb::launch_finalize(natoms * nframes, natoms, reinterpret_cast<const dpb::ForceSum *>(acc), force, atom_energy,
                              nullptr, atom_energy, energy, nframes, pos, nullptr, err, status,
                              (cudaStream_t)stream);
}

// Kernels of the curl-SVD transforms and of the fncB operator.
//
// fncB (reference: fun_Lanczos/fncB.m:3-6) on a quasi-periodic n^3 grid is
//   y = blkdiag(Pr, Qr)^H * [M J^H; J N] * blkdiag(Pr, Qr) * x
// with Pr = Psi*Pi.Pr, Qr = Phi*Pi.Qr (Funhand_Generate_Lanzcos.m:79-82) and
// Psi = Phi = S .* unitary-inverse-DFT per component (gMtxVecMul_FFT.m:10-36).
// The Bloch phase S is diagonal and the interpolated material operators are
// built from Bloch shifts T_d, so S^H T_d S = tau_d P_d with P_d the periodic
// shift and tau_d = exp(i theta_d / n).  fncB therefore runs entirely in the
// periodic frame: S is never applied, and every shift carries the constant
// phase tau_d.
//
// Material operators (IntCovarForm{N_vertex,M_vertex_new,J_vertex_new}.m and
// the symmetrisation in Interpolation_Material_Matrix_Mult_Point_vertex.m:22-26)
// factor into  edge/face -> vertex gathers, a per-vertex 3x3 tensor product,
// and vertex -> edge/face scatters:
//   U_j = 1/4 (I+T_a)^H (I+T_b)^H u_j   (a, b = axes != j)   face -> vertex
//   V_j = 1/2 (I+T_j)^H v_j                                  edge -> vertex
//   Hu_i = sum_{j!=i} Mh_ij U_j + sum_j conj(J_ji) V_j
//   Hv_i = sum_{j!=i} Nh_ij V_j + sum_j J_ij U_j
//   u'_i = m_i u_i + 1/4 (I+T_a)(I+T_b) Hu_i ,  m_i = face average of Re Mh_ii
//   v'_i = n_i v_i + 1/2 (I+T_i) Hv_i        ,  n_i = edge average of Re Nh_ii
// where Mh, Nh are the Hermitian parts of the vertex tensors: (X + X^H)/2 of
// the assembled operator equals the operator built from Herm(A).
//
// Pipeline (one launch each):
//   plane_inv  : Pi blocks per frequency voxel + inverse DFT along x and y
//   col        : inverse DFT along z (in place)
//   sweep      : u', v' in one pass into the second buffer (fncb_material.cuh),
//                or the two-kernel form: vertex (U, V, Hu, Hv at every vertex
//                into scratch) then faceedge (u', v' in place)
//   col        : forward DFT along z
//   plane_fwd  : forward DFT along y and x + Pi^H blocks
//
// This header holds the size-templated kernels; fncb_inst_*.cu instantiate
// them per precision and grid size so the size list compiles in parallel,
// and fncb_stencil.cu holds the size-independent kernels and the dispatch.
#pragma once

#include "fame_internal.h"
#include "fft_reg.cuh"
#include "fncb_material.cuh"

namespace fame {
namespace detail {


constexpr double kInvSqrt14 = 0.26726124191242438468455348087975;

template <class R> struct PiBlock {
  cx<R> p1[3], p2[3];
  R sig;
};

// SVD_Matrix_curl.m:45-57 for one frequency voxel: with L = (Lx, Ly, Lz),
// w = (1,2,3)/sqrt(14):  Pi1 = (conj(L) x w)/|conj(L) x w|,
// Pi2 = (conj(Pi1) x conj(L))/|L|, Sigma = |L|.
template <class R>
__device__ __forceinline__ PiBlock<R> pi_block(cx<R> lx, cx<R> ly, cx<R> lz) {
  const R w1 = R(1 * kInvSqrt14), w2 = R(2 * kInvSqrt14), w3 = R(3 * kInvSqrt14);
  R lq = lx.x * lx.x + lx.y * lx.y + ly.x * ly.x + ly.y * ly.y + lz.x * lz.x + lz.y * lz.y;
  cx<R> lw = mk<R>(w1 * lx.x + w2 * ly.x + w3 * lz.x, w1 * lx.y + w2 * ly.y + w3 * lz.y);
  R n1sq = lq - (lw.x * lw.x + lw.y * lw.y);
  R inv1 = rsqrt(n1sq);
  R inv0 = rsqrt(lq);
  R sq = lq * inv0;
  cx<R> b0 = cconj(lx), b1 = cconj(ly), b2 = cconj(lz);
  PiBlock<R> P;
  P.p1[0] = cscale(csub(cscale(b1, w3), cscale(b2, w2)), inv1);
  P.p1[1] = cscale(csub(cscale(b2, w1), cscale(b0, w3)), inv1);
  P.p1[2] = cscale(csub(cscale(b0, w2), cscale(b1, w1)), inv1);
  cx<R> c0 = cconj(P.p1[0]), c1 = cconj(P.p1[1]), c2 = cconj(P.p1[2]);
  P.p2[0] = cscale(csub(cmul(c1, b2), cmul(c2, b1)), inv0);
  P.p2[1] = cscale(csub(cmul(c2, b0), cmul(c0, b2)), inv0);
  P.p2[2] = cscale(csub(cmul(c0, b1), cmul(c1, b0)), inv0);
  P.sig = sq;
  return P;
}

// Pi1 | Pi2 of one voxel from the plan's table (6 complex; three 16-byte
// loads in complex64).
template <class R>
__device__ __forceinline__ PiBlock<R> pi_load(const cx<R>* p) {
  PiBlock<R> P;
  if constexpr (sizeof(R) == 4) {
    const float4* q = reinterpret_cast<const float4*>(p);
    const float4 a = __ldg(q), b = __ldg(q + 1), c = __ldg(q + 2);
    P.p1[0] = mk<R>(a.x, a.y);
    P.p1[1] = mk<R>(a.z, a.w);
    P.p1[2] = mk<R>(b.x, b.y);
    P.p2[0] = mk<R>(b.z, b.w);
    P.p2[1] = mk<R>(c.x, c.y);
    P.p2[2] = mk<R>(c.z, c.w);
  } else if constexpr (std::is_same<R, double>::value) {
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      P.p1[i] = __ldg(p + i);
      P.p2[i] = __ldg(p + 3 + i);
    }
  } else {
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      P.p1[i] = p[i];
      P.p2[i] = p[3 + i];
    }
  }
  P.sig = R(0);
  return P;
}

// Pi of voxel (i1, i2, k3) of instance inst: from the table when the plan has
// one (voxel index k3*N*N + e, e = i2*N + i1), else evaluated.
template <class R, int N>
__device__ __forceinline__ PiBlock<R> pi_at(const PlanData<R>& d, int inst, int k3, int e, const cx<R>* lam, int i1,
                                            int i2, cx<R> lz) {
  if (d.pi) return pi_load<R>(d.pi + ((size_t)inst * N * N * N + (size_t)k3 * N * N + e) * 6);
  return pi_block<R>(lam[i1], lam[N + i2], lz);
}

// Pi of the voxels of one frequency plane (k3 fixed) in complex64, where the
// plane kernels evaluate it.  With m = L x w (w = (1,2,3)/sqrt(14)) and
// q = m x conj(L):
//   Pi1 = conj(m)/|m|,  Pi2 = q/(|m| |L|),
// and m_0, m_1, their products with conj(L) and the squared norms depend on
// one of (i2, k3), (i1, k3) only: a row table in shared memory (PiRow) and
// registers of a thread that stays in one column (PiCol) hold them, which
// leaves 16 operations and two reciprocal square roots per voxel before the
// products with the vectors (the blocks took about 100, 40 % of the kernels'
// instructions; at n = 60, 10 vectors, k_plane_inv 26.3 -> 19.4 M warp
// instructions, 58 -> 47 us).  |m|^2 as a sum of squares also has no
// cancellation: fncB's error against 64 bits 3.5e-7 -> 2.2e-7.
//
// Side 0 (Pr) takes the same formulas with conj(L) for L and the two blocks
// swapped:  side 1: v = conj(m) X + q Y with X = a/|m|, Y = b/(|m||L|);
//           side 0: the same with X = b/|m|, Y = -a/(|m||L|).
struct PiRow {
  float2 ly, m0, t1, t2;  // L_y, m_0, m_0 conj(L_z), m_0 conj(L_y)
  float lq, n1;           // |L_y|^2, |m_0|^2
  float2 pad;
};
struct PiCol {
  float2 w2lx, lx, m1, k1, k2;  // w_2 L_x, L_x, m_1, m_1 conj(L_z), m_1 conj(L_x)
  float lq, n1;                 // |L_x|^2 + |L_z|^2, |m_1|^2
};
struct PiVox {
  float2 m0, m1, m2, q0, q1, q2;
  float inv1, i01;  // 1/|m|, 1/(|m||L|)
};
__device__ __forceinline__ float2 side_conj(float2 v, int side) { return side ? v : cconj(v); }
template <int N>
__device__ __forceinline__ void pi_row_fill(PiRow* rows, const float2* lam, int k3, int side, int i2) {
  const float2 lz = side_conj(lam[2 * N + k3], side), ly = side_conj(lam[N + i2], side);
  const float w2 = float(2 * kInvSqrt14), w3 = float(3 * kInvSqrt14);
  PiRow r;
  r.ly = ly;
  r.m0 = caxpy(-w2, lz, cscale(ly, w3));
  r.t1 = cmulc(lz, r.m0);
  r.t2 = cmulc(ly, r.m0);
  r.lq = ly.x * ly.x + ly.y * ly.y;
  r.n1 = r.m0.x * r.m0.x + r.m0.y * r.m0.y;
  r.pad = make_float2(0.f, 0.f);
  rows[i2] = r;
}
template <int N> __device__ __forceinline__ PiCol pi_col(const float2* lam, int k3, int side, int i1) {
  const float2 lz = side_conj(lam[2 * N + k3], side);
  const float w1 = float(1 * kInvSqrt14), w2 = float(2 * kInvSqrt14), w3 = float(3 * kInvSqrt14);
  PiCol c;
  c.lx = side_conj(lam[i1], side);
  c.w2lx = cscale(c.lx, w2);
  c.m1 = caxpy(-w3, c.lx, cscale(lz, w1));
  c.k1 = cmulc(lz, c.m1);
  c.k2 = cmulc(c.lx, c.m1);
  c.lq = c.lx.x * c.lx.x + c.lx.y * c.lx.y + lz.x * lz.x + lz.y * lz.y;
  c.n1 = c.m1.x * c.m1.x + c.m1.y * c.m1.y;
  return c;
}
__device__ __forceinline__ PiVox pi_vox(const PiRow* row, const PiCol& c) {
  const float4* q = reinterpret_cast<const float4*>(row);
  const float4 a = q[0], b = q[1], n = q[2];
  const float2 ly = make_float2(a.x, a.y), t1 = make_float2(b.x, b.y), t2 = make_float2(b.z, b.w);
  PiVox v;
  v.m0 = make_float2(a.z, a.w);
  v.m1 = c.m1;
  v.m2 = caxpy(-float(kInvSqrt14), ly, c.w2lx);
  v.q0 = csub(c.k1, cmulc(ly, v.m2));
  v.q1 = csub(cmulc(c.lx, v.m2), t1);
  v.q2 = csub(t2, c.k2);
  const float n1 = fmaf(v.m2.x, v.m2.x, fmaf(v.m2.y, v.m2.y, n.y + c.n1));
  v.inv1 = rsqrtf(n1);
  v.i01 = v.inv1 * rsqrtf(n.x + c.lq);
  return v;
}
// (a, b) of one side -> the three frequency components (Pi.Pr / Pi.Qr)
__device__ __forceinline__ void pi_prep(const PiVox& P, int side, float2 a, float2 b, float sc, float2 (&v)[3]) {
  const float s1 = P.inv1 * sc, s2 = P.i01 * sc;
  const float2 X = cscale(side ? a : b, s1), Y = cscale(side ? b : a, side ? s2 : -s2);
  v[0] = cfma(P.q0, Y, cmulc(P.m0, X));
  v[1] = cfma(P.q1, Y, cmulc(P.m1, X));
  v[2] = cfma(P.q2, Y, cmulc(P.m2, X));
}
// the adjoint: three components -> (a, b)
__device__ __forceinline__ void pi_post(const PiVox& P, int side, const float2 (&u)[3], float sc, float2& a, float2& b) {
  const float s1 = P.inv1 * sc, s2 = P.i01 * sc;
  const float2 X = cscale(cfma(P.m2, u[2], cfma(P.m1, u[1], cmul(P.m0, u[0]))), s1);
  const float2 Y = cscale(cfmac(P.q2, u[2], cfmac(P.q1, u[1], cmulc(P.q0, u[0]))), side ? s2 : -s2);
  a = side ? X : Y;
  b = side ? Y : X;
}

// Bytes of shared memory of the plane kernels: three padded fields, and the
// row table in complex64.
template <class R, int N> constexpr size_t plane_smem() {
  return sizeof(cx<R>) * 3 * N * (N + 1) + (sizeof(R) == 4 ? sizeof(PiRow) * N : 0);
}
// The row table's place behind the fields (16-byte aligned: N is even).
template <class R, int N> __device__ __forceinline__ PiRow* pi_rows(cx<R>* sm) {
  return reinterpret_cast<PiRow*>(sm + 3 * N * (N + 1));
}

// Scale of a unitary 3D DFT, n^{-3/2}.  The S-free transforms of fncB put all of
// it on the plane kernels' frequency side (two blocks per voxel and side), so
// the z pass multiplies by nothing.
template <class R, int N> __device__ __forceinline__ R scale3() {
  constexpr double s = 1.0 / (double(N) * csqrt_int(N));
  return R(s);
}

// Operator input / output of the split plane kernels.  The double-single
// operator reads and writes complex128 vectors (the caller's), converting
// on load and store, so it needs no conversion passes; the conversions run
// on the FP64 pipe, which its float-float arithmetic leaves idle.
template <class R> __device__ __forceinline__ cx<R> load_io(const cx<R>* p) {
  if constexpr (std::is_same<R, ff>::value) {
    const double2 v = *reinterpret_cast<const double2*>(p);
    cff c;
    c.x = ff(v.x);
    c.y = ff(v.y);
    return c;
  } else {
    return *p;
  }
}
template <class R> __device__ __forceinline__ void store_io(cx<R>* p, cx<R> v) {
  if constexpr (std::is_same<R, ff>::value) {
    *reinterpret_cast<double2*>(p) = make_double2(double(v.x), double(v.y));
  } else {
    *p = v;
  }
}

// The conjugate-gradient direction update p = z + beta p, done by the first
// kernel of fncB on the p it reads (z == null: no update).  Each CTA rewrites
// the plane of p it loads, so the separate update pass over p disappears.
template <class R> struct DirUpd {
  const cx<R>* z = nullptr;     // same layout and strides as p
  const double* beta = nullptr; // [nvec] of this launch
};

// ---------------------------------------------------------------------------
// plane_inv: one CTA per (k3 plane, side, vector); 3N threads.
// PREP: build the 3 frequency components of one side from (a, b):
//   side 0 (Pr):  p = -conj(Pi2) a + conj(Pi1) b      (Pi.Pr, SVD_Matrix_curl.m:64)
//   side 1 (Qr):  q =  Pi1 a + Pi2 b                  (Pi.Qr, SVD_Matrix_curl.m:63)
// else copy 3 components.  Then inverse DFT along x (rows, via shared
// memory) and y (columns, straight to global); WITH_S multiplies by S_x S_y / n
// there, PREP without S scales its input by n^{-3/2} (scale3).
// ---------------------------------------------------------------------------
template <class R, int N, bool PREP, bool WITH_S>
__global__ void __launch_bounds__(((3 * N + 31) / 32) * 32, sizeof(R) == 4 ? 2 : 1)
k_plane_inv(const cx<R>* __restrict__ x, cx<R>* __restrict__ out, PlanData<R> d, VecCtx ctx,
            long long in_stride, long long in_side_stride, long long out_stride, int side0, DirUpd<R> upd) {
  constexpr int LD = N + 1;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cx<R>* sm = reinterpret_cast<cx<R>*>(smem_raw);  // [3][N][LD]
  const int k3 = blockIdx.x;
  const int vec = blockIdx.z;
  if (ctx.active && !ctx.active[vec]) return;
  const int inst = vec_inst(ctx, vec);
  const int side = side0 + blockIdx.y;
  const long long Nq = (long long)N * N * N;
  const cx<R>* lam = d.lam + (long long)inst * 3 * N;
  const cx<R>* xin = x + vec * in_stride + blockIdx.y * in_side_stride + (long long)k3 * N * N;
  const int tid = threadIdx.x;

  // Input plane -> shared memory: thread (column i1, row group) takes rows
  // grp, grp + 3, ...  The global loads of PF rows are issued together before
  // any is used, so a CTA waits for one memory round trip per batch.
  constexpr bool PIV = PREP && sizeof(R) == 4;
  const int grp = tid / N, i1 = tid - grp * N;
  const bool act = tid < 3 * N;
  if constexpr (PIV) {
    if (tid < N) pi_row_fill<N>(pi_rows<R, N>(sm), lam, k3, side, tid);
  }
  constexpr int ITEMS = (N + 2) / 3;
  constexpr int NB = PREP ? 2 : 3;                        // input blocks
  constexpr int PF0 = (sizeof(R) == 4 ? 24 : 12) / NB;   // rows in flight per thread
  constexpr int NBATCH = (ITEMS + PF0 - 1) / PF0;
  constexpr int PF = (ITEMS + NBATCH - 1) / NBATCH;
  static_for<0, NBATCH>([&](auto bc) {
    constexpr int base = decltype(bc)::value * PF;
    cx<R> in[PF][NB];
#pragma unroll
    for (int it = 0; it < PF; ++it) {
      const int i2 = grp + 3 * (base + it);
      if (act && i2 < N) {
#pragma unroll
        for (int c = 0; c < NB; ++c) in[it][c] = xin[c * Nq + i2 * N + i1];
      }
    }
    if (PREP && upd.z) {  // p = z + beta p, written back
      const long long off = vec * in_stride + blockIdx.y * in_side_stride + (long long)k3 * N * N;
      const cx<R>* zin = upd.z + off;
      cx<R>* xw = const_cast<cx<R>*>(x) + off;
      const R bt = R(upd.beta[vec]);
      cx<R> zz[PF][NB];
#pragma unroll
      for (int it = 0; it < PF; ++it) {
        const int i2 = grp + 3 * (base + it);
        if (act && i2 < N) {
#pragma unroll
          for (int c = 0; c < NB; ++c) zz[it][c] = zin[c * Nq + i2 * N + i1];
        }
      }
#pragma unroll
      for (int it = 0; it < PF; ++it) {
        const int i2 = grp + 3 * (base + it);
        if (act && i2 < N) {
#pragma unroll
          for (int c = 0; c < NB; ++c) {
            in[it][c] = caxpy(bt, in[it][c], zz[it][c]);
            xw[c * Nq + i2 * N + i1] = in[it][c];
          }
        }
      }
    }
    if constexpr (PIV && decltype(bc)::value == 0) __syncthreads();  // the row table
    if (act) {
      if constexpr (PIV) {
        const PiCol pc = pi_col<N>(lam, k3, side, i1);
#pragma unroll
        for (int it = 0; it < PF; ++it) {
          const int i2 = grp + 3 * (base + it);
          if (i2 < N) {
            cx<R> v[3];
            pi_prep(pi_vox(pi_rows<R, N>(sm) + i2, pc), side, in[it][0], in[it][1],
                    WITH_S ? R(1) : scale3<R, N>(), v);
#pragma unroll
            for (int c = 0; c < 3; ++c) sm[(c * N + i2) * LD + i1] = v[c];
          }
        }
      } else {
#pragma unroll
        for (int it = 0; it < PF; ++it) {
          const int i2 = grp + 3 * (base + it);
          if (i2 < N) {
            cx<R> v0, v1, v2;
            if constexpr (PREP) {
              PiBlock<R> P = pi_at<R, N>(d, inst, k3, i2 * N + i1, lam, i1, i2, lam[2 * N + k3]);
              cx<R> a = in[it][0], b = in[it][1];
              if constexpr (!WITH_S) {
                a = cscale(a, scale3<R, N>());
                b = cscale(b, scale3<R, N>());
              }
              if (side == 0) {
                v0 = cfmac(P.p1[0], b, cneg(cmulc(P.p2[0], a)));
                v1 = cfmac(P.p1[1], b, cneg(cmulc(P.p2[1], a)));
                v2 = cfmac(P.p1[2], b, cneg(cmulc(P.p2[2], a)));
              } else {
                v0 = cfma(P.p2[0], b, cmul(P.p1[0], a));
                v1 = cfma(P.p2[1], b, cmul(P.p1[1], a));
                v2 = cfma(P.p2[2], b, cmul(P.p1[2], a));
              }
            } else {
              v0 = in[it][0];
              v1 = in[it][1];
              v2 = in[it][NB - 1];
            }
            sm[(0 * N + i2) * LD + i1] = v0;
            sm[(1 * N + i2) * LD + i1] = v1;
            sm[(2 * N + i2) * LD + i1] = v2;
          }
        }
      }
    }
  });
  __syncthreads();
  if (tid < 3 * N) {  // x rows
    const int c = tid / N, i2 = tid - c * N;
    cx<R>* row = sm + (c * N + i2) * LD;
    cx<R> v[N];
#pragma unroll
    for (int i = 0; i < N; ++i) v[i] = row[i];
    fft<R, N, +1>(v);
#pragma unroll
    for (int i = 0; i < N; ++i) row[i] = v[i];
  }
  __syncthreads();
  if (tid < 3 * N) {  // y columns
    const int c = tid / N, i1 = tid - c * N;
    cx<R> v[N];
#pragma unroll
    for (int i = 0; i < N; ++i) v[i] = sm[(c * N + i) * LD + i1];
    fft<R, N, +1>(v);
    cx<R> sx = mk<R>(R(1), R(0));
    const cx<R>* S = d.sxyz + (long long)inst * 3 * N;
    if constexpr (WITH_S) sx = cscale(S[i1], R(1.0 / N));
    cx<R>* o = out + vec * out_stride + (long long)(blockIdx.y * 3 + c) * Nq + (long long)k3 * N * N + i1;
#pragma unroll
    for (int i2 = 0; i2 < N; ++i2) {
      cx<R> r = v[i2];
      if constexpr (WITH_S) r = cmul(r, cmul(sx, S[N + i2]));
      o[(long long)i2 * N] = r;
    }
  }
}

// ---------------------------------------------------------------------------
// plane_fwd: one CTA per (k3 plane, side, vector); 3N threads.
// Forward DFT along y (columns, straight from global) and x (rows, shared
// memory); WITH_S multiplies conj(S_x S_y) / n first.  POST applies
// the Pi^H blocks of one side (SVD_Matrix_curl.m:63-64, handles Prs/Qrs):
//   side 0 (Prs): a = -sum_c Pi2_c u_c,  b = sum_c Pi1_c u_c
//   side 1 (Qrs): a = sum_c conj(Pi1_c) v_c, b = sum_c conj(Pi2_c) v_c
// else copies the 3 components out.
// ---------------------------------------------------------------------------
template <class R, int N, bool POST, bool WITH_S>
__global__ void __launch_bounds__(((3 * N + 31) / 32) * 32, sizeof(R) == 4 ? 2 : 1)
k_plane_fwd(const cx<R>* __restrict__ w, cx<R>* __restrict__ y, PlanData<R> d, VecCtx ctx,
            long long w_stride, long long out_stride, long long out_side_stride, int side0) {
  constexpr int LD = N + 1;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cx<R>* sm = reinterpret_cast<cx<R>*>(smem_raw);  // [3][N][LD]
  const int k3 = blockIdx.x;
  const int vec = blockIdx.z;
  if (ctx.active && !ctx.active[vec]) return;
  const int inst = vec_inst(ctx, vec);
  const int side = side0 + blockIdx.y;
  const long long Nq = (long long)N * N * N;
  const int tid = threadIdx.x;
  const cx<R>* S = d.sxyz + (long long)inst * 3 * N;
  const cx<R>* lam = d.lam + (long long)inst * 3 * N;
  if constexpr (POST && sizeof(R) == 4) {
    if (tid < N) pi_row_fill<N>(pi_rows<R, N>(sm), lam, k3, side, tid);
  }
  if (tid < 3 * N) {  // y columns
    const int c = tid / N, i1 = tid - c * N;
    const cx<R>* src = w + vec * w_stride + (long long)(blockIdx.y * 3 + c) * Nq + (long long)k3 * N * N + i1;
    cx<R> v[N];
    cx<R> sx = mk<R>(R(1), R(0));
    if constexpr (WITH_S) sx = cscale(S[i1], R(1.0 / N));
#pragma unroll
    for (int i2 = 0; i2 < N; ++i2) {
      v[i2] = src[(long long)i2 * N];
      if constexpr (WITH_S) v[i2] = cmulc(cmul(sx, S[N + i2]), v[i2]);
    }
    fft<R, N, -1>(v);
#pragma unroll
    for (int i2 = 0; i2 < N; ++i2) sm[(c * N + i2) * LD + i1] = v[i2];
  }
  __syncthreads();
  if (tid < 3 * N) {  // x rows
    const int c = tid / N, i2 = tid - c * N;
    cx<R>* row = sm + (c * N + i2) * LD;
    cx<R> v[N];
#pragma unroll
    for (int i = 0; i < N; ++i) v[i] = row[i];
    fft<R, N, -1>(v);
#pragma unroll
    for (int i = 0; i < N; ++i) row[i] = v[i];
  }
  __syncthreads();
  cx<R>* o = y + vec * out_stride + blockIdx.y * out_side_stride + (long long)k3 * N * N;
  if (tid < 3 * N) {
    const int grp = tid / N, i1 = tid - grp * N;
    if constexpr (POST && sizeof(R) == 4) {
      const PiCol pc = pi_col<N>(lam, k3, side, i1);
#pragma unroll 4
      for (int i2 = grp; i2 < N; i2 += 3) {
        const cx<R> u[3] = {sm[(0 * N + i2) * LD + i1], sm[(1 * N + i2) * LD + i1], sm[(2 * N + i2) * LD + i1]};
        cx<R> a, b;
        pi_post(pi_vox(pi_rows<R, N>(sm) + i2, pc), side, u, WITH_S ? R(1) : scale3<R, N>(), a, b);
        o[i2 * N + i1] = a;
        o[Nq + i2 * N + i1] = b;
      }
    } else {
#pragma unroll 4
      for (int i2 = grp; i2 < N; i2 += 3) {
        const int e = i2 * N + i1;
        cx<R> u0 = sm[(0 * N + i2) * LD + i1];
        cx<R> u1 = sm[(1 * N + i2) * LD + i1];
        cx<R> u2 = sm[(2 * N + i2) * LD + i1];
        if constexpr (POST) {
          PiBlock<R> P = pi_at<R, N>(d, inst, k3, e, lam, i1, i2, lam[2 * N + k3]);
          cx<R> a, b;
          if (side == 0) {
            a = cneg(cfma(P.p2[2], u2, cfma(P.p2[1], u1, cmul(P.p2[0], u0))));
            b = cfma(P.p1[2], u2, cfma(P.p1[1], u1, cmul(P.p1[0], u0)));
          } else {
            a = cfmac(P.p1[2], u2, cfmac(P.p1[1], u1, cmulc(P.p1[0], u0)));
            b = cfmac(P.p2[2], u2, cfmac(P.p2[1], u1, cmulc(P.p2[0], u0)));
          }
          if constexpr (!WITH_S) {
            a = cscale(a, scale3<R, N>());
            b = cscale(b, scale3<R, N>());
          }
          o[e] = a;
          o[Nq + e] = b;
        } else {
          o[e] = u0;
          o[Nq + e] = u1;
          o[2 * Nq + e] = u2;
        }
      }
    }
  }
}

// ---------------------------------------------------------------------------
// Split-pencil plane kernels of fncB (k_plane_inv2 / k_plane_fwd2): the same
// work as k_plane_inv<PREP> / k_plane_fwd<POST>, with G threads per pencil
// instead of one.  A length N = G*M with gcd(G, M) = 1 is split by the
// prime-factor index map (no twiddle factors):
//   n = (M*n1 + G*n2) mod N,  k = (M*A*k1 + G*B*k2) mod N,
//   A = M^{-1} mod G, B = G^{-1} mod M,
//   X[k] = sum_{n2} W_M^{n2 k2} sum_{n1} x[n] W_G^{n1 k1}.
// Pass A: M length-G DFTs over n1 per pencil, in place in shared memory
// (thread g of the pencil takes n2 = g, g+G, ...).  Pass B: thread k1 takes
// the length-M DFT over n2 in registers.  A thread then holds M complex
// values instead of N, so 3*N*G threads of a CTA fit two CTAs per SM
// (N = 60: G = 3, 540 threads, 34 warps per SM against 12 for one thread per
// 60-point pencil).
// ---------------------------------------------------------------------------

// CTAs per SM the split kernels are compiled for: two for the default lane
// count in complex64, one otherwise (the register allocation then decides).
template <class R, int N, int G> constexpr int plane_min_blocks() {
  return sizeof(R) == 4 && G == plane_split(N) ? 2 : 1;
}

template <int N, int G> struct Split {
  static constexpr int M = N / G;
  static constexpr int A = fft_inv_mod(M % G, G);
  static constexpr int B = fft_inv_mod(G % M, M);
  static constexpr int T = 3 * N * G;                 // threads: (field, pencil, g)
  static constexpr int TB = ((T + 31) / 32) * 32;
  static constexpr int NA = (M + G - 1) / G;          // pass-A DFTs per thread (upper bound)
  static_assert(G * M == N && A >= 0 && B >= 0, "coprime split");
  FAME_HD static constexpr int in_slot(int n1, int n2) { return (M * n1 + G * n2) % N; }
  FAME_HD static constexpr int out_slot(int k1, int k2) { return (M * A * k1 + G * B * k2) % N; }
};

// Pass A on one pencil in shared memory (element i at p[i * STRIDE]) for the
// thread with sub-pencil index GC (compile time, so that every slot index is
// an immediate offset).
template <class R, int N, int G, int S, int STRIDE, int GC>
__device__ __forceinline__ void split_pass_a(cx<R>* p) {
  using SP = Split<N, G>;
  static_for<0, SP::NA>([&](auto jc) {
    constexpr int n2 = GC + decltype(jc)::value * G;
    if constexpr (n2 < SP::M) {
      cx<R> a[G];
      static_for<0, G>([&](auto n1c) { a[decltype(n1c)::value] = p[SP::in_slot(decltype(n1c)::value, n2) * STRIDE]; });
      fft<R, G, S>(a);
      static_for<0, G>([&](auto n1c) { p[SP::in_slot(decltype(n1c)::value, n2) * STRIDE] = a[decltype(n1c)::value]; });
    }
  });
}

// Pass B read: the M values of row K1 of one pencil.
template <class R, int N, int G, int STRIDE, int K1>
__device__ __forceinline__ void split_pass_b_load(const cx<R>* p, cx<R> (&z)[N / G]) {
  using SP = Split<N, G>;
  static_for<0, SP::M>([&](auto n2c) { z[decltype(n2c)::value] = p[SP::in_slot(K1, decltype(n2c)::value) * STRIDE]; });
}

// Pass B write: X[out_slot(K1, k2)] = z[k2].
template <class R, int N, int G, int STRIDE, int K1, class P>
__device__ __forceinline__ void split_pass_b_store(P p, const cx<R> (&z)[N / G]) {
  using SP = Split<N, G>;
  static_for<0, SP::M>([&](auto k2c) { p[(long long)SP::out_slot(K1, decltype(k2c)::value) * STRIDE] = z[decltype(k2c)::value]; });
}

// f(integral_constant<GC>) for the runtime g of this thread (warps are
// uniform in g except the ones that straddle two sub-pencil groups).
template <int G, class F> __device__ __forceinline__ void with_g(int g, F&& f) {
  static_for<0, G>([&](auto gc) {
    if (g == decltype(gc)::value) f(gc);
  });
}

template <class R, int N, int G, bool UPD>
__global__ void __launch_bounds__(Split<N, G>::TB, plane_min_blocks<R, N, G>())
k_plane_inv2(const cx<R>* __restrict__ x, cx<R>* __restrict__ out, PlanData<R> d, VecCtx ctx,
             long long in_stride, long long in_side_stride, long long out_stride, int side0, DirUpd<R> upd) {
  using SP = Split<N, G>;
  constexpr int M = SP::M, T = SP::T, LD = N + 1;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cx<R>* sm = reinterpret_cast<cx<R>*>(smem_raw);  // [3][N][LD]
  const int k3 = blockIdx.x;
  const int vec = blockIdx.z;
  if (ctx.active && !ctx.active[vec]) return;
  const int inst = vec_inst(ctx, vec);
  const int side = side0 + blockIdx.y;
  const long long Nq = (long long)N * N * N;
  const cx<R>* lam = d.lam + (long long)inst * 3 * N;
  const cx<R>* xin = x + vec * in_stride + blockIdx.y * in_side_stride + (long long)k3 * N * N;
  const int tid = threadIdx.x;
  // Pi blocks (frequency voxel -> 3 components of this side), scaled for the
  // three inverse DFTs: thread (column i1, row group) takes every NG-th row;
  // all loads of a thread issued together.
  {
    constexpr int NG = 3 * G;
    constexpr int ITEMS = (N + NG - 1) / NG;
    const int grp = tid / N, i1 = tid - grp * N;
    if constexpr (sizeof(R) == 4) {
      if (tid < N) pi_row_fill<N>(pi_rows<R, N>(sm), lam, k3, side, tid);
    }
    cx<R> in[ITEMS][2];
#pragma unroll
    for (int it = 0; it < ITEMS; ++it) {
      const int i2 = grp + it * NG;
      if (tid < T && i2 < N) {
        in[it][0] = load_io<R>(xin + i2 * N + i1);
        in[it][1] = load_io<R>(xin + Nq + i2 * N + i1);
      }
    }
    if constexpr (UPD) {  // p = z + beta p, written back (UPD: upd.z set)
      const long long off = vec * in_stride + blockIdx.y * in_side_stride + (long long)k3 * N * N;
      const cx<R>* zin = upd.z + off;
      cx<R>* xw = const_cast<cx<R>*>(x) + off;
      const R bt = R(upd.beta[vec]);
#pragma unroll
      for (int it = 0; it < ITEMS; ++it) {
        const int i2 = grp + it * NG;
        if (tid < T && i2 < N) {
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            in[it][c] = caxpy(bt, in[it][c], zin[c * Nq + i2 * N + i1]);
            xw[c * Nq + i2 * N + i1] = in[it][c];
          }
        }
      }
    }
    const R sc = scale3<R, N>();
    if constexpr (sizeof(R) == 4) {
      __syncthreads();  // the row table
      if (tid < T) {
        const PiCol pc = pi_col<N>(lam, k3, side, i1);
#pragma unroll
        for (int it = 0; it < ITEMS; ++it) {
          const int i2 = grp + it * NG;
          if (i2 < N) {
            cx<R> v[3];
            pi_prep(pi_vox(pi_rows<R, N>(sm) + i2, pc), side, in[it][0], in[it][1], sc, v);
#pragma unroll
            for (int c = 0; c < 3; ++c) sm[(c * N + i2) * LD + i1] = v[c];
          }
        }
      }
    } else {
      const cx<R> lz = lam[2 * N + k3];
#pragma unroll
      for (int it = 0; it < ITEMS; ++it) {
        const int i2 = grp + it * NG;
        if (tid < T && i2 < N) {
          PiBlock<R> P = pi_at<R, N>(d, inst, k3, i2 * N + i1, lam, i1, i2, lz);
          const cx<R> a = cscale(in[it][0], sc), b = cscale(in[it][1], sc);
          cx<R> v0, v1, v2;
          if (side == 0) {
            v0 = cfmac(P.p1[0], b, cneg(cmulc(P.p2[0], a)));
            v1 = cfmac(P.p1[1], b, cneg(cmulc(P.p2[1], a)));
            v2 = cfmac(P.p1[2], b, cneg(cmulc(P.p2[2], a)));
          } else {
            v0 = cfma(P.p2[0], b, cmul(P.p1[0], a));
            v1 = cfma(P.p2[1], b, cmul(P.p1[1], a));
            v2 = cfma(P.p2[2], b, cmul(P.p1[2], a));
          }
          sm[(0 * N + i2) * LD + i1] = v0;
          sm[(1 * N + i2) * LD + i1] = v1;
          sm[(2 * N + i2) * LD + i1] = v2;
        }
      }
    }
  }
  __syncthreads();
  const int g = tid / (3 * N);
  const int cp = tid - g * (3 * N);
  const int c = cp / N, p = cp - c * N;
  const bool act = tid < T;
  // x rows (pencil p = row i2 of field c)
  if (act) with_g<G>(g, [&](auto gc) { split_pass_a<R, N, G, +1, 1, decltype(gc)::value>(sm + (c * N + p) * LD); });
  __syncthreads();
  {
    cx<R> z[M];
    if (act)
      with_g<G>(g, [&](auto gc) { split_pass_b_load<R, N, G, 1, decltype(gc)::value>(sm + (c * N + p) * LD, z); });
    if (act) fft<R, M, +1>(z);
    __syncthreads();
    if (act)
      with_g<G>(g, [&](auto gc) { split_pass_b_store<R, N, G, 1, decltype(gc)::value>(sm + (c * N + p) * LD, z); });
  }
  __syncthreads();
  // y columns (pencil p = column i1 of field c), written straight to global
  if (act) with_g<G>(g, [&](auto gc) { split_pass_a<R, N, G, +1, LD, decltype(gc)::value>(sm + c * N * LD + p); });
  __syncthreads();
  if (act) {
    cx<R> z[M];
    with_g<G>(g, [&](auto gc) { split_pass_b_load<R, N, G, LD, decltype(gc)::value>(sm + c * N * LD + p, z); });
    fft<R, M, +1>(z);
    cx<R>* o = out + vec * out_stride + (long long)(blockIdx.y * 3 + c) * Nq + (long long)k3 * N * N + p;
    with_g<G>(g, [&](auto gc) { split_pass_b_store<R, N, G, N, decltype(gc)::value>(o, z); });
  }
}

template <class R, int N, int G>
__global__ void __launch_bounds__(Split<N, G>::TB, plane_min_blocks<R, N, G>())
k_plane_fwd2(const cx<R>* __restrict__ w, cx<R>* __restrict__ y, PlanData<R> d, VecCtx ctx,
             long long w_stride, long long out_stride, long long out_side_stride, int side0) {
  using SP = Split<N, G>;
  constexpr int M = SP::M, T = SP::T, LD = N + 1;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cx<R>* sm = reinterpret_cast<cx<R>*>(smem_raw);  // [3][N][LD]
  const int k3 = blockIdx.x;
  const int vec = blockIdx.z;
  if (ctx.active && !ctx.active[vec]) return;
  const int inst = vec_inst(ctx, vec);
  const int side = side0 + blockIdx.y;
  const long long Nq = (long long)N * N * N;
  const int tid = threadIdx.x;
  const int g = tid / (3 * N);
  const int cp = tid - g * (3 * N);
  const int c = cp / N, p = cp - c * N;
  const bool act = tid < T;
  const cx<R>* lam = d.lam + (long long)inst * 3 * N;
  if constexpr (sizeof(R) == 4) {
    if (tid < N) pi_row_fill<N>(pi_rows<R, N>(sm), lam, k3, side, tid);
  }
  // y columns, pass A straight from global (pencil p = column i1 of field c)
  if (act) {
    const cx<R>* src = w + vec * w_stride + (long long)(blockIdx.y * 3 + c) * Nq + (long long)k3 * N * N + p;
    cx<R>* col = sm + c * N * LD + p;
    with_g<G>(g, [&](auto gc) {
      constexpr int GC = decltype(gc)::value;
      cx<R> a[SP::NA][G];
      static_for<0, SP::NA>([&](auto jc) {
        constexpr int n2 = GC + decltype(jc)::value * G;
        if constexpr (n2 < M)
          static_for<0, G>([&](auto n1c) {
            a[decltype(jc)::value][decltype(n1c)::value] = src[(long long)SP::in_slot(decltype(n1c)::value, n2) * N];
          });
      });
      static_for<0, SP::NA>([&](auto jc) {
        constexpr int j = decltype(jc)::value;
        constexpr int n2 = GC + j * G;
        if constexpr (n2 < M) {
          fft<R, G, -1>(a[j]);
          static_for<0, G>([&](auto n1c) { col[SP::in_slot(decltype(n1c)::value, n2) * LD] = a[j][decltype(n1c)::value]; });
        }
      });
    });
  }
  __syncthreads();
  {
    cx<R> z[M];
    if (act)
      with_g<G>(g, [&](auto gc) { split_pass_b_load<R, N, G, LD, decltype(gc)::value>(sm + c * N * LD + p, z); });
    if (act) fft<R, M, -1>(z);
    __syncthreads();
    if (act)
      with_g<G>(g, [&](auto gc) { split_pass_b_store<R, N, G, LD, decltype(gc)::value>(sm + c * N * LD + p, z); });
  }
  __syncthreads();
  // x rows (pencil p = row i2 of field c)
  if (act) with_g<G>(g, [&](auto gc) { split_pass_a<R, N, G, -1, 1, decltype(gc)::value>(sm + (c * N + p) * LD); });
  __syncthreads();
  {
    cx<R> z[M];
    if (act)
      with_g<G>(g, [&](auto gc) { split_pass_b_load<R, N, G, 1, decltype(gc)::value>(sm + (c * N + p) * LD, z); });
    if (act) fft<R, M, -1>(z);
    __syncthreads();
    if (act)
      with_g<G>(g, [&](auto gc) { split_pass_b_store<R, N, G, 1, decltype(gc)::value>(sm + (c * N + p) * LD, z); });
  }
  __syncthreads();
  // Pi^H blocks of this side, scaled for the three forward DFTs
  cx<R>* o = y + vec * out_stride + blockIdx.y * out_side_stride + (long long)k3 * N * N;
  const R sc = scale3<R, N>();
  if (!act) return;
  const int grp = tid / N, i1 = tid - grp * N;
  if constexpr (sizeof(R) == 4) {
    const PiCol pc = pi_col<N>(lam, k3, side, i1);
#pragma unroll 2
    for (int i2 = grp; i2 < N; i2 += 3 * G) {
      const cx<R> u[3] = {sm[(0 * N + i2) * LD + i1], sm[(1 * N + i2) * LD + i1], sm[(2 * N + i2) * LD + i1]};
      cx<R> a, b;
      pi_post(pi_vox(pi_rows<R, N>(sm) + i2, pc), side, u, sc, a, b);
      o[i2 * N + i1] = a;
      o[Nq + i2 * N + i1] = b;
    }
  } else {
    const cx<R> lz = lam[2 * N + k3];
    for (int i2 = grp; i2 < N; i2 += 3 * G) {
      const int e = i2 * N + i1;
      const cx<R> u0 = sm[(0 * N + i2) * LD + i1];
      const cx<R> u1 = sm[(1 * N + i2) * LD + i1];
      const cx<R> u2 = sm[(2 * N + i2) * LD + i1];
      PiBlock<R> P = pi_at<R, N>(d, inst, k3, e, lam, i1, i2, lz);
      cx<R> a, b;
      if (side == 0) {
        a = cneg(cfma(P.p2[2], u2, cfma(P.p2[1], u1, cmul(P.p2[0], u0))));
        b = cfma(P.p1[2], u2, cfma(P.p1[1], u1, cmul(P.p1[0], u0)));
      } else {
        a = cfmac(P.p1[2], u2, cfmac(P.p1[1], u1, cmulc(P.p1[0], u0)));
        b = cfmac(P.p2[2], u2, cfmac(P.p2[1], u1, cmulc(P.p2[0], u0)));
      }
      store_io<R>(o + e, cscale(a, sc));
      store_io<R>(o + Nq + e, cscale(b, sc));
    }
  }
}

// ---------------------------------------------------------------------------
// col: DFT along z of every (i1, i2) column, in place; one thread per column.
// SMODE 1: multiply S_z(i3) after (inverse); 2: multiply conj(S_z(i3)) before
// (forward), both scaled by 1/sqrt(n); 0: neither (scale3).
// ---------------------------------------------------------------------------
template <class R, int N, int DIR, int SMODE>
__global__ void __launch_bounds__(128, sizeof(R) == 4 ? 3 : 1)
k_col(cx<R>* __restrict__ w, PlanData<R> d, VecCtx ctx, long long stride) {
  const int col = blockIdx.x * blockDim.x + threadIdx.x;
  const int f = blockIdx.y;
  const int vec = blockIdx.z;
  if (col >= N * N) return;
  if (ctx.active && !ctx.active[vec]) return;
  const long long Nq = (long long)N * N * N;
  cx<R>* p = w + vec * stride + (long long)f * Nq + col;
  const cx<R>* Sz = d.sxyz + (long long)vec_inst(ctx, vec) * 3 * N + 2 * N;
  cx<R> v[N];
#pragma unroll
  for (int i = 0; i < N; ++i) {
    v[i] = p[(long long)i * N * N];
    if constexpr (SMODE == 2) v[i] = cmulc(Sz[i], v[i]);
  }
  fft<R, N, DIR>(v);
  constexpr double scale = 1.0 / csqrt_int(N);
#pragma unroll
  for (int i = 0; i < N; ++i) {
    cx<R> r = v[i];
    if constexpr (SMODE != 0) r = cscale(r, R(scale));
    if constexpr (SMODE == 1) r = cmul(Sz[i], r);
    p[(long long)i * N * N] = r;
  }
}

inline dim3 grid_pts(long long Nq, int nvec, int tpb) {
  return dim3((unsigned)((Nq + tpb - 1) / tpb), (unsigned)nvec, 1);
}

// Lanes per pencil of the split plane kernels for a tuned value (< 0: the
// default of size N; 0: one thread per pencil) under the plan's option;
// a count not compiled for N falls back to the default.
template <class R, int N> inline int plane_lanes(const Plan& P, int tuned) {
  if (std::is_same<R, ff>::value && (tuned == 0 || !P.opt_plane_split)) tuned = -1;  // double-single: split only
  else if (!P.opt_plane_split || plane_split(N) == 0 || tuned == 0) return 0;
  for (int i = 0; i < kPlaneLanesMax; ++i)
    if (tuned > 0 && plane_lanes_alt(N, i) == tuned) return tuned;
  return plane_split(N);
}

// The split an untuned fncB of nvec vectors takes (as a tuned value).  In
// complex64: one thread per pencil once the 2 N nvec CTAs give every SM its
// two resident ones (it needs a quarter fewer instructions and half the
// shared-memory traffic: fncB of 4 vectors at n = 40 60 -> 50 us, 8 at n = 48
// 116 -> 106, 10 at n = 60 260 -> 246), the size's split below that, where
// the extra warps hide latency (one vector at n = 48 41.5 -> 37.5 us, n = 60
// 52 -> 49).  nvec is the whole batch, so sub-batches do not change a result.
template <class R, int N> inline int default_lanes(const Plan& P, int nvec) {
  return std::is_same<R, float>::value && N * nvec >= P.sms ? 0 : -1;
}

// f(integral_constant<G>) for the compiled lane count G == lanes of size N.
template <class R, int N, class F> inline void with_lanes(int lanes, F&& f) {
  static_assert(kPlaneLanesMax == 3, "one branch per compiled lane count");
  constexpr int g0 = plane_lanes_alt(N, 0), g1 = plane_lanes_alt(N, 1), g2 = plane_lanes_alt(N, 2);
  if constexpr (g0 > 0)
    if (lanes == g0) return f(std::integral_constant<int, g0>{});
  if constexpr (g1 > 0)
    if (lanes == g1) return f(std::integral_constant<int, g1>{});
  if constexpr (g2 > 0)
    if (lanes == g2) return f(std::integral_constant<int, g2>{});
}

template <class R, int N, bool PREP, bool WITH_S>
cudaError_t plane_inv(const Plan& P, const PlanData<R>& d, const cx<R>* x, cx<R>* out, int nvec,
                      int nside, int side0, long long in_stride, long long in_side_stride,
                      long long out_stride, const VecCtx& ctx, cudaStream_t st, DirUpd<R> upd = DirUpd<R>(),
                      int tuned_lanes = -1) {
  constexpr size_t sm = plane_smem<R, N>();
  if constexpr (PREP && !WITH_S && plane_split(N) > 0) {
    const int lanes = plane_lanes<R, N>(P, tuned_lanes);
    if (lanes > 0) {
      cudaError_t e = cudaErrorInvalidValue;
      // the CG direction update is compiled into its own variant, so the
      // plain operator carries none of its code (the double-single operator
      // never takes it)
      auto launch = [&](auto kfn, int tb) {
        e = cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
        if (e != cudaSuccess) return;
        FAME_LAUNCHED(1);
        kfn<<<dim3(N, nside, nvec), tb, sm, st>>>(x, out, d, ctx, in_stride, in_side_stride, out_stride, side0, upd);
        e = cudaGetLastError();
      };
      with_lanes<R, N>(lanes, [&](auto gc) {
        constexpr int G = decltype(gc)::value;
        if constexpr (!std::is_same<R, ff>::value) {
          if (upd.z) return launch(k_plane_inv2<R, N, G, true>, Split<N, G>::TB);
        }
        launch(k_plane_inv2<R, N, G, false>, Split<N, G>::TB);
      });
      return e;
    }
  }
  if constexpr (std::is_same<R, ff>::value && PREP && !WITH_S && plane_split(N) > 0) {
    return cudaErrorInvalidValue;  // double-single: split kernels only (above)
  } else {
    const int threads = ((3 * N + 31) / 32) * 32;
    auto kfn = k_plane_inv<R, N, PREP, WITH_S>;
    cudaError_t e = cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    if (e != cudaSuccess) return e;
    FAME_LAUNCHED(1);
    kfn<<<dim3(N, nside, nvec), threads, sm, st>>>(x, out, d, ctx, in_stride, in_side_stride, out_stride,
                                                   side0, upd);
    return cudaGetLastError();
  }
}

template <class R, int N, bool POST, bool WITH_S>
cudaError_t plane_fwd(const Plan& P, const PlanData<R>& d, const cx<R>* w, cx<R>* y, int nvec, int nside,
                      int side0, long long w_stride, long long out_stride, long long out_side_stride,
                      const VecCtx& ctx, cudaStream_t st, int tuned_lanes = -1) {
  constexpr size_t sm = plane_smem<R, N>();
  if constexpr (POST && !WITH_S && plane_split(N) > 0) {
    const int lanes = plane_lanes<R, N>(P, tuned_lanes);
    if (lanes > 0) {
      cudaError_t e = cudaErrorInvalidValue;
      with_lanes<R, N>(lanes, [&](auto gc) {
        constexpr int G = decltype(gc)::value;
        auto kfn = k_plane_fwd2<R, N, G>;
        e = cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
        if (e != cudaSuccess) return;
        FAME_LAUNCHED(1);
        kfn<<<dim3(N, nside, nvec), Split<N, G>::TB, sm, st>>>(w, y, d, ctx, w_stride, out_stride,
                                                               out_side_stride, side0);
        e = cudaGetLastError();
      });
      return e;
    }
  }
  if constexpr (std::is_same<R, ff>::value && POST && !WITH_S && plane_split(N) > 0) {
    return cudaErrorInvalidValue;  // double-single: split kernels only (above)
  } else {
    const int threads = ((3 * N + 31) / 32) * 32;
    auto kfn = k_plane_fwd<R, N, POST, WITH_S>;
    cudaError_t e = cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    if (e != cudaSuccess) return e;
    FAME_LAUNCHED(1);
    kfn<<<dim3(N, nside, nvec), threads, sm, st>>>(w, y, d, ctx, w_stride, out_stride, out_side_stride,
                                                   side0);
    return cudaGetLastError();
  }
}

// ---------------------------------------------------------------------------
// col2: the z-DFT with the same prime-factor split as the plane kernels, for
// the double-single type (one thread holding a whole 60-point column of
// float-float pairs needs 240 registers of data alone).  One CTA per
// (y row, field, vector): the row's N columns (all z) are staged in shared
// memory with coalesced row loads, G threads per column do the length-G
// passes in place, then each the length-M DFT of its sub-pencil in
// registers, written straight back to global (consecutive threads hold
// consecutive x).  No scale (scale3), no S multiply.
// ---------------------------------------------------------------------------
template <class R, int N, int DIR>
__global__ void __launch_bounds__(((N * plane_split(N) + 31) / 32) * 32)
k_col2(cx<R>* __restrict__ w, VecCtx ctx, long long stride) {
  constexpr int G = plane_split(N);
  using SP = Split<N, G>;
  constexpr int M = SP::M, LD = N + 1, T = N * G;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cx<R>* sm = reinterpret_cast<cx<R>*>(smem_raw);  // [z][LD]
  const int y = blockIdx.x;
  const int vec = blockIdx.z;
  if (ctx.active && !ctx.active[vec]) return;
  const long long NN = (long long)N * N;
  cx<R>* base = w + vec * stride + (long long)blockIdx.y * N * NN + (long long)y * N;
  const int tid = threadIdx.x;
  for (int e = tid; e < N * N; e += blockDim.x) {
    const int z = e / N, x = e - z * N;
    sm[z * LD + x] = base[(long long)z * NN + x];
  }
  __syncthreads();
  const int g = tid / N, p = tid - g * N;
  const bool act = tid < T;
  if (act) with_g<G>(g, [&](auto gc) { split_pass_a<R, N, G, DIR, LD, decltype(gc)::value>(sm + p); });
  __syncthreads();
  if (act) {
    cx<R> z[M];
    with_g<G>(g, [&](auto gc) { split_pass_b_load<R, N, G, LD, decltype(gc)::value>(sm + p, z); });
    fft<R, M, DIR>(z);
    with_g<G>(g, [&](auto gc) { split_pass_b_store<R, N, G, (int)(N * N), decltype(gc)::value>(base + p, z); });
  }
}

template <class R, int N, int DIR, int SMODE>
cudaError_t col(const Plan& P, const PlanData<R>& d, cx<R>* w, int nfield, int nvec, long long stride, const VecCtx& ctx,
                cudaStream_t st) {
  if constexpr (std::is_same<R, ff>::value && SMODE == 0 && plane_split(N) > 0) {
    constexpr int G = plane_split(N);
    const size_t sm = sizeof(cx<R>) * N * (N + 1);
    auto kfn = k_col2<R, N, DIR>;
    cudaError_t e = cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    if (e != cudaSuccess) return e;
    FAME_LAUNCHED(1);
    kfn<<<dim3(N, nfield, nvec), ((N * G + 31) / 32) * 32, sm, st>>>(w, ctx, stride);
    return cudaGetLastError();
  } else {
    // One warp per CTA in complex128 and for small complex64 batches: the work
    // of a launch is then spread over the SMs warp by warp (two vectors at
    // n = 30 are 96 CTAs of four warps, up to four warps on an SM where the
    // even share is 2.2: 23 -> 16 us), 128 threads where there are plenty.
    const int tpb = sizeof(R) == 8 || (long long)N * N * nfield * nvec < 128LL * 6 * P.sms ? 32 : 128;
    dim3 g((N * N + tpb - 1) / tpb, nfield, nvec);
    FAME_LAUNCHED(1);
    k_col<R, N, DIR, SMODE><<<g, tpb, 0, st>>>(w, d, ctx, stride);
    return cudaGetLastError();
  }
}


// fncB on a batch, as sub-batches of `chunk` vectors (0: all at once) so that
// the six-field intermediates of a sub-batch can stay in L2; the stencil
// kernels run with tpb threads per block.  Both come from fame_autotune.
//
// pq (may be null): with the single-pass stencil, per-CTA partial sums of
// Re(x^H B x) (sweep_partials_n per vector, vector-major).  The curl-SVD
// transforms are unitary and Pi has orthonormal columns, so x^H B x equals
// w^H [M J^H; J N] w for the spatial fields w the stencil reads; the stencil
// pass accumulates it while it writes its output.
//
// pupd_z / pupd_beta (may be null): x is a CG direction p, updated first as
// p = z + beta p (in place) by the plane kernel that reads it.
template <class R, int N>
cudaError_t fncB_n(const Plan& P, const cx<R>* x, cx<R>* y, int nvec, const VecCtx& ctx, cx<R>* w0, cx<R>* w1,
                   cudaStream_t st, double2* pq, const cx<R>* pupd_z, const double* pupd_beta) {
  static_assert(!std::is_same<R, ff>::value || plane_split(N) > 0,
                "the double-single fncB reads and writes complex128 through the split plane kernels");
  PlanData<R> d = pdata<R>(P);
  if (!P.opt_pi_table) d.pi = nullptr;  // evaluate Pi in the plane kernels instead
  const long long Nq = P.Nq;
  const TuneEntry tn = tune_for(P, tune_prec<R>(), nvec);
  const int chunk = sub_batch(tn, nvec);
  const int tz = sweep_planes<R, N>(P, chunk);
  const int lanes = tn.lanes >= 0 ? tn.lanes : default_lanes<R, N>(P, nvec);
  for (int v0 = 0; v0 < nvec; v0 += chunk) {
    const int nv = std::min(chunk, nvec - v0);
    const VecCtx c = sub_ctx(ctx, v0);
    const cx<R>* xs = x + (size_t)v0 * 4 * Nq;
    cx<R>* ys = y + (size_t)v0 * 4 * Nq;
    cudaError_t e;
    DirUpd<R> upd;
    if (pupd_z) {
      upd.z = pupd_z + (size_t)v0 * 4 * Nq;
      upd.beta = pupd_beta + v0;
    }
    e = plane_inv<R, N, true, false>(P, d, xs, w0, nv, 2, 0, 4 * Nq, 2 * Nq, 6 * Nq, c, st, upd, lanes);
    if (e != cudaSuccess) return e;
    e = col<R, N, +1, 0>(P, d, w0, 6, nv, 6 * Nq, c, st);
    if (e != cudaSuccess) return e;
    // material stencil: single pass w0 -> w1, or the two-kernel form in place on w0
    cx<R>* wm = w0;
    if (tn.stencil_tpb == 0) {
      e = sweep_n<R, N>(P, w0, w1, nv, c, st, tz, pq ? pq + (size_t)v0 * sweep_partials_n<R, N>(tz) : nullptr);
      wm = w1;
    } else {
      e = stencil_n<R, N>(P, w0, w0, w1, nv, c, st, tn.stencil_tpb, false);
    }
    if (e != cudaSuccess) return e;
    e = col<R, N, -1, 0>(P, d, wm, 6, nv, 6 * Nq, c, st);
    if (e != cudaSuccess) return e;
    e = plane_fwd<R, N, true, false>(P, d, wm, ys, nv, 2, 0, 6 * Nq, 4 * Nq, 2 * Nq, c, st, lanes);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

template <class R, int N>
cudaError_t fields_inv_n(const Plan& P, const cx<R>* x, cx<R>* w, int nvec, const VecCtx& ctx, cudaStream_t st) {
  const PlanData<R>& d = pdata<R>(P);
  const long long Nq = P.Nq;
  cudaError_t e = plane_inv<R, N, true, false>(P, d, x, w, nvec, 2, 0, 4 * Nq, 2 * Nq, 6 * Nq, ctx, st);
  if (e != cudaSuccess) return e;
  return col<R, N, +1, 0>(P, d, w, 6, nvec, 6 * Nq, ctx, st);
}

template <class R, int N>
cudaError_t transform_n(const Plan& P, int trans, const cx<R>* x, cx<R>* y, int nvec, const VecCtx& ctx,
                        cudaStream_t st) {
  const PlanData<R>& d = pdata<R>(P);
  const long long Nq = P.Nq;
  cudaError_t e;
  if (trans == 0) {
    e = plane_inv<R, N, false, true>(P, d, x, y, nvec, 1, 0, 3 * Nq, 0, 3 * Nq, ctx, st);
    if (e != cudaSuccess) return e;
    return col<R, N, +1, 1>(P, d, y, 3, nvec, 3 * Nq, ctx, st);
  }
  // transpose: z first (conj(S_z) before), then y, x with conj(S_x S_y) before.
  if (x != y) {
    e = cudaMemcpyAsync(y, x, sizeof(cx<R>) * 3 * Nq * nvec, cudaMemcpyDeviceToDevice, st);
    if (e != cudaSuccess) return e;
  }
  e = col<R, N, -1, 2>(P, d, y, 3, nvec, 3 * Nq, ctx, st);
  if (e != cudaSuccess) return e;
  return plane_fwd<R, N, false, true>(P, d, y, y, nvec, 1, 0, 3 * Nq, 3 * Nq, 0, ctx, st);
}

template <class R, int N>
cudaError_t handle_n(const Plan& P, int which, const cx<R>* x, cx<R>* y, int nvec, const VecCtx& ctx,
                     cx<R>* w0, cudaStream_t st) {
  const PlanData<R>& d = pdata<R>(P);
  const long long Nq = P.Nq;
  cudaError_t e;
  if (which == 0 || which == 1) {  // Pr / Qr : 2Nq -> 3Nq
    e = plane_inv<R, N, true, true>(P, d, x, y, nvec, 1, which, 2 * Nq, 0, 3 * Nq, ctx, st);
    if (e != cudaSuccess) return e;
    return col<R, N, +1, 1>(P, d, y, 3, nvec, 3 * Nq, ctx, st);
  }
  // Prs / Qrs : 3Nq -> 2Nq through the 3Nq scratch w0
  e = cudaMemcpyAsync(w0, x, sizeof(cx<R>) * 3 * Nq * nvec, cudaMemcpyDeviceToDevice, st);
  if (e != cudaSuccess) return e;
  e = col<R, N, -1, 2>(P, d, w0, 3, nvec, 3 * Nq, ctx, st);
  if (e != cudaSuccess) return e;
  return plane_fwd<R, N, true, true>(P, d, w0, y, nvec, 1, which - 2, 3 * Nq, 2 * Nq, 0, ctx, st);
}


}  // namespace detail
}  // namespace fame

// Declarations of the size-templated entry points of one (precision, size),
// each prefixed by PFX ("template" to instantiate, "extern template" to
// suppress instantiation in other translation units).
#define FAME_SIZE_SIGS(PFX, R, NN)                                                                                 \
  PFX cudaError_t fame::detail::fncB_n<R, NN>(const Plan&, const cx<R>*, cx<R>*, int, const VecCtx&, cx<R>*,       \
                                              cx<R>*, cudaStream_t, double2*, const cx<R>*, const double*);       \
  PFX cudaError_t fame::detail::stencil_n<R, NN>(const Plan&, const cx<R>*, cx<R>*, cx<R>*, int, const VecCtx&,    \
                                                 cudaStream_t, int, bool);                                         \
  PFX cudaError_t fame::detail::fields_inv_n<R, NN>(const Plan&, const cx<R>*, cx<R>*, int, const VecCtx&,         \
                                                    cudaStream_t);                                                 \
  PFX cudaError_t fame::detail::transform_n<R, NN>(const Plan&, int, const cx<R>*, cx<R>*, int, const VecCtx&,     \
                                                   cudaStream_t);                                                  \
  PFX cudaError_t fame::detail::handle_n<R, NN>(const Plan&, int, const cx<R>*, cx<R>*, int, const VecCtx&,        \
                                                cx<R>*, cudaStream_t);
// explicit instantiation of one (precision, size)
#define FAME_INST_SIZE(R, NN) FAME_SIZE_SIGS(template, R, NN)

// Grid sizes with a compiled double-single fncB (the residuals b - B x of the
// mixed inner solves; other sizes take the FP64 fncB), and its declaration.
// (sizes with a split of the plane kernels: their loads and stores convert the
// complex128 vectors; at n = 32 the unsplit double-single kernels were no
// faster than FP64)
#define FAME_FOR_EACH_DS_N(X) X(12) X(24) X(40) X(48) X(60)
#define FAME_DS_SIGS(PFX, NN)                                                                                      \
  PFX cudaError_t fame::detail::fncB_n<fame::ff, NN>(const Plan&, const cx<fame::ff>*, cx<fame::ff>*, int,         \
                                                     const VecCtx&, cx<fame::ff>*, cx<fame::ff>*, cudaStream_t,    \
                                                     double2*, const cx<fame::ff>*, const double*);
#define FAME_INST_DS(NN) FAME_DS_SIGS(template, NN)

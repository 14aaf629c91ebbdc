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
//                (complex64: k_plane_inv, three fields of a plane per CTA;
//                complex128 and double-single: k_field_inv, one field)
//   col        : inverse DFT along z (in place)
//   sweep      : u', v' in one pass into the second buffer (fncb_material.cuh),
//                or the two-kernel form: vertex (U, V, Hu, Hv at every vertex
//                into scratch) then faceedge (u', v' in place)
//   col        : forward DFT along z
//   plane_fwd  : forward DFT along y and x + Pi^H blocks (k_plane_fwd, k_field_fwd)
// The curl transforms and the handles use the same kernels; S is applied in
// the z pass.
//
// This header holds the size-templated kernels; fncb_inst_*.cu instantiate
// them per precision and grid size so the size list compiles in parallel,
// and fncb_stencil.cu holds the size-independent kernels and the dispatch.
#pragma once

#include <cooperative_groups.h>

#include "fame_internal.h"
#include "fft_reg.cuh"
#include "launch.h"
#include "fncb_material.cuh"

namespace fame {
namespace detail {


constexpr double kInvSqrt14 = 0.26726124191242438468455348087975;

// conj(v) if keep is 0, v otherwise, by the sign bits (no arithmetic).
__device__ __forceinline__ double2 conj_unless(double2 v, int keep) {
  const int m = keep ? 0 : (int)0x80000000;
  return make_double2(v.x, __hiloint2double(__double2hiint(v.y) ^ m, __double2loint(v.y)));
}
__device__ __forceinline__ cff conj_unless(cff v, int keep) {
  const int m = keep ? 0 : (int)0x80000000;
  v.y = ff(__int_as_float(__float_as_int(v.y.hi) ^ m), __int_as_float(__float_as_int(v.y.lo) ^ m), true);
  return v;
}

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

// Scale of a unitary 3D DFT, n^{-3/2}.  Pi carries all of it (two blocks per
// voxel and side), so neither the plane kernels nor the z pass multiply by it.
template <class R, int N> __device__ __forceinline__ R scale3() {
  constexpr double s = 1.0 / (double(N) * csqrt_int(N));
  return R(s);
}

// Component c of Pi1 and Pi2 at a frequency voxel (index vox = k3 n^2 + i2 n +
// i1) of instance inst, times n^{-3/2}: from the plan's table [6][n^3], or
// (pi_comp) evaluated when there is none.
template <class R> struct PiComp {
  cx<R> p1, p2;
};
template <class R, int N>
__device__ __forceinline__ PiComp<R> pi_table(const PlanData<R>& d, int inst, int c, int vox) {
  constexpr int Nq = N * N * N;
  const cx<R>* t = d.pi + (size_t)inst * 6 * Nq + vox;
  PiComp<R> P;
  P.p1 = t[(size_t)c * Nq];
  P.p2 = t[(size_t)(3 + c) * Nq];
  return P;
}
template <class R, int N>
__device__ __forceinline__ PiComp<R> pi_comp(const PlanData<R>& d, int inst, int c, int vox, const cx<R>* lam) {
  PiComp<R> P;
  if (d.pi) {
    P = pi_table<R, N>(d, inst, c, vox);
  } else {
    const PiBlock<R> B = pi_block<R>(lam[vox % N], lam[N + (vox / N) % N], lam[2 * N + vox / (N * N)]);
    P.p1 = cscale(c == 0 ? B.p1[0] : c == 1 ? B.p1[1] : B.p1[2], scale3<R, N>());
    P.p2 = cscale(c == 0 ? B.p2[0] : c == 1 ? B.p2[1] : B.p2[2], scale3<R, N>());
  }
  return P;
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
// cancellation where L is nearly parallel to w, which |L|^2 - |L.w|^2 has:
// fncB's error against 64 bits 3.5e-7 -> 2.2e-7 of the norm, its worst element
// (220 batches at n = 40 to 64) 3.3e-4 -> 1.6e-6.
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

// Bytes of shared memory of the complex64 plane kernels: three padded fields
// and the row table.
template <int N> constexpr size_t plane_smem() { return sizeof(float2) * 3 * N * (N + 1) + sizeof(PiRow) * N; }
// The row table's place behind the fields (16-byte aligned: N is even).
template <int N> __device__ __forceinline__ PiRow* pi_rows(float2* sm) {
  return reinterpret_cast<PiRow*>(sm + 3 * N * (N + 1));
}

// Operator input / output of the field kernels.  The double-single
// operator reads and writes complex128 vectors (the caller's), converting
// on load and store, so it needs no conversion passes; by bit operations, as
// an FP64 or conversion instruction takes as long as 64 FP32 ones.
// The element type that the caller's vectors have.
template <class R> using io_t = std::conditional_t<std::is_same_v<R, ff>, double2, cx<R>>;
template <class R> __device__ __forceinline__ io_t<R> load_raw(const cx<R>* p) {
  return *reinterpret_cast<const io_t<R>*>(p);
}
template <class R> __device__ __forceinline__ cx<R> from_io(io_t<R> v) {
  if constexpr (std::is_same<R, ff>::value) {
    cff c;
    const bool ok = ff_split_bits(__double2hiint(v.x), __double2loint(v.x), c.x) &
                    ff_split_bits(__double2hiint(v.y), __double2loint(v.y), c.y);
    if (__any_sync(__activemask(), !ok)) {  // a branch of the whole warp, so that the FP64 form costs nothing elsewhere
      c.x = ff(v.x);
      c.y = ff(v.y);
    }
    return c;
  } else {
    return v;
  }
}
template <class R> __device__ __forceinline__ cx<R> load_io(const cx<R>* p) { return from_io<R>(load_raw<R>(p)); }
template <class R> __device__ __forceinline__ void store_io(cx<R>* p, cx<R> v) {
  if constexpr (std::is_same<R, ff>::value) {
    uint32_t h[4], l[4];
    const bool ok = f32_widen_bits(v.x.hi, h[0], l[0]) & f32_widen_bits(v.x.lo, h[1], l[1]) &
                    f32_widen_bits(v.y.hi, h[2], l[2]) & f32_widen_bits(v.y.lo, h[3], l[3]);
    double2 o = make_double2(__hiloint2double(h[0], l[0]) + __hiloint2double(h[1], l[1]),
                             __hiloint2double(h[2], l[2]) + __hiloint2double(h[3], l[3]));
    if (__any_sync(__activemask(), !ok)) o = make_double2(double(v.x), double(v.y));
    *reinterpret_cast<double2*>(p) = o;
  } else {
    *p = v;
  }
}

// ---------------------------------------------------------------------------
// complex64 plane kernels: one CTA per (k3 plane, side, vector), 3N threads,
// one thread per pencil (N <= 64 complex values in registers).
//
// k_plane_inv: PREP builds the three frequency components of one side from
// (a, b), else it copies three components; then the inverse DFT along x
// (rows, via shared memory) and y (columns, straight to global).
//   side 0 (Pr):  p = -conj(Pi2) a + conj(Pi1) b      (Pi.Pr, SVD_Matrix_curl.m:64)
//   side 1 (Qr):  q =  Pi1 a + Pi2 b                  (Pi.Qr, SVD_Matrix_curl.m:63)
// Latency-bound: at n = 60 two CTAs of six warps fit an SM (88 KB of shared
// memory each) and issue 40 % of the cycles.  A prime-factor split of each
// pencil over three threads (34 warps per SM) needed twice the shared-memory
// traffic and a third more instructions, and was slower at every size and
// batch (n = 60, warm, one vector 9.4 against 8.6 us, ten 58 against 47).
// ---------------------------------------------------------------------------
template <int N, bool PREP>
__global__ void __launch_bounds__(((3 * N + 31) / 32) * 32, 2)
k_plane_inv(const float2* __restrict__ x, float2* __restrict__ out, PlanData<float> d,
            const __grid_constant__ VecCtx ctx, long long in_stride, long long in_side_stride,
            long long out_stride, int side0) {
  constexpr int LD = N + 1;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float2* sm = reinterpret_cast<float2*>(smem_raw);  // [3][N][LD]
  const int k3 = blockIdx.x;
  const int vec = blockIdx.z;
  const int inst = vec_inst(ctx, vec);
  const int side = side0 + blockIdx.y;
  const long long Nq = (long long)N * N * N;
  const float2* lam = d.lam + (long long)inst * 3 * N;
  const long long off = vec * in_stride + blockIdx.y * in_side_stride + (long long)k3 * N * N;
  const float2* xin = x + off;
  const int tid = threadIdx.x;

  // Input plane -> shared memory: thread (column i1, row group) takes rows
  // grp, grp + 3, ...  The global loads of PF rows are issued together before
  // any is used, so a CTA waits for one memory round trip per batch.
  const int grp = tid / N, i1 = tid - grp * N;
  const bool act = tid < 3 * N;
  if constexpr (PREP) {  // plan tables only: before the wait
    if (tid < N) pi_row_fill<N>(pi_rows<N>(sm), lam, k3, side, tid);
  }
  pdl_wait();
  if (ctx.active && !ctx.active[vec]) return;
  constexpr int ITEMS = (N + 2) / 3;
  constexpr int NB = PREP ? 2 : 3;                        // input blocks
  constexpr int NBATCH = (ITEMS * NB + 23) / 24;
  constexpr int PF = (ITEMS + NBATCH - 1) / NBATCH;       // rows in flight per thread
  static_for<0, NBATCH>([&](auto bc) {
    constexpr int base = decltype(bc)::value * PF;
    float2 in[PF][NB];
#pragma unroll
    for (int it = 0; it < PF; ++it) {
      const int i2 = grp + 3 * (base + it);
      if (act && i2 < N) {
#pragma unroll
        for (int c = 0; c < NB; ++c) in[it][c] = xin[c * Nq + i2 * N + i1];
      }
    }
    if constexpr (PREP && decltype(bc)::value == 0) __syncthreads();  // the row table
    if (act) {
      [[maybe_unused]] PiCol pc;
      if constexpr (PREP) pc = pi_col<N>(lam, k3, side, i1);
#pragma unroll
      for (int it = 0; it < PF; ++it) {
        const int i2 = grp + 3 * (base + it);
        if (i2 < N) {
          float2 v[3];
          if constexpr (PREP) {
            pi_prep(pi_vox(pi_rows<N>(sm) + i2, pc), side, in[it][0], in[it][1], scale3<float, N>(), v);
          } else {
#pragma unroll
            for (int c = 0; c < 3; ++c) v[c] = in[it][c < NB ? c : 0];
          }
#pragma unroll
          for (int c = 0; c < 3; ++c) sm[(c * N + i2) * LD + i1] = v[c];
        }
      }
    }
  });
  __syncthreads();
  if (act) {  // x rows
    float2* row = sm + tid * LD;
    float2 v[N];
#pragma unroll
    for (int i = 0; i < N; ++i) v[i] = row[i];
    fft<float, N, +1>(v);
#pragma unroll
    for (int i = 0; i < N; ++i) row[i] = v[i];
  }
  __syncthreads();
  if (act) {  // y columns (field grp, column i1)
    float2 v[N];
#pragma unroll
    for (int i = 0; i < N; ++i) v[i] = sm[(grp * N + i) * LD + i1];
    fft<float, N, +1>(v);
    float2* o = out + vec * out_stride + (long long)(blockIdx.y * 3 + grp) * Nq + (long long)k3 * N * N + i1;
#pragma unroll
    for (int i2 = 0; i2 < N; ++i2) o[(long long)i2 * N] = v[i2];
  }
}

// k_plane_fwd: forward DFT along y (columns, straight from global) and x
// (rows, shared memory).  POST applies the Pi^H blocks of one side
// (SVD_Matrix_curl.m:63-64, handles Prs/Qrs):
//   side 0 (Prs): a = -sum_c Pi2_c u_c,  b = sum_c Pi1_c u_c
//   side 1 (Qrs): a = sum_c conj(Pi1_c) v_c, b = sum_c conj(Pi2_c) v_c
// else copies the 3 components out.
template <int N, bool POST>
__global__ void __launch_bounds__(((3 * N + 31) / 32) * 32, 2)
k_plane_fwd(const float2* __restrict__ w, float2* __restrict__ y, PlanData<float> d, const __grid_constant__ VecCtx ctx,
            long long w_stride, long long out_stride, long long out_side_stride, int side0) {
  constexpr int LD = N + 1;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float2* sm = reinterpret_cast<float2*>(smem_raw);  // [3][N][LD]
  const int k3 = blockIdx.x;
  const int vec = blockIdx.z;
  const int inst = vec_inst(ctx, vec);
  const int side = side0 + blockIdx.y;
  const long long Nq = (long long)N * N * N;
  const int tid = threadIdx.x;
  const int grp = tid / N, i1 = tid - grp * N;
  const bool act = tid < 3 * N;
  const float2* lam = d.lam + (long long)inst * 3 * N;
  if constexpr (POST) {
    if (tid < N) pi_row_fill<N>(pi_rows<N>(sm), lam, k3, side, tid);
  }
  pdl_wait();
  if (ctx.active && !ctx.active[vec]) return;
  if (act) {  // y columns (field grp, column i1)
    const float2* src = w + vec * w_stride + (long long)(blockIdx.y * 3 + grp) * Nq + (long long)k3 * N * N + i1;
    float2 v[N];
#pragma unroll
    for (int i2 = 0; i2 < N; ++i2) v[i2] = src[(long long)i2 * N];
    fft<float, N, -1>(v);
#pragma unroll
    for (int i2 = 0; i2 < N; ++i2) sm[(grp * N + i2) * LD + i1] = v[i2];
  }
  __syncthreads();
  if (act) {  // x rows
    float2* row = sm + tid * LD;
    float2 v[N];
#pragma unroll
    for (int i = 0; i < N; ++i) v[i] = row[i];
    fft<float, N, -1>(v);
#pragma unroll
    for (int i = 0; i < N; ++i) row[i] = v[i];
  }
  __syncthreads();
  if (!act) return;
  float2* o = y + vec * out_stride + blockIdx.y * out_side_stride + (long long)k3 * N * N;
  [[maybe_unused]] PiCol pc;
  if constexpr (POST) pc = pi_col<N>(lam, k3, side, i1);
#pragma unroll 4
  for (int i2 = grp; i2 < N; i2 += 3) {
    const float2 u[3] = {sm[(0 * N + i2) * LD + i1], sm[(1 * N + i2) * LD + i1], sm[(2 * N + i2) * LD + i1]};
    const int e = i2 * N + i1;
    if constexpr (POST) {
      float2 a, b;
      pi_post(pi_vox(pi_rows<N>(sm) + i2, pc), side, u, scale3<float, N>(), a, b);
      o[e] = a;
      o[Nq + e] = b;
    } else {
#pragma unroll
      for (int c = 0; c < 3; ++c) o[c * Nq + e] = u[c];
    }
  }
}

// ---------------------------------------------------------------------------
// complex128 and double-single field kernels: the same work, one CTA per
// (k3 plane, field, vector), so that the arithmetic of a launch spreads over
// the SMs in thirds of a plane.  (With the three fields in one CTA, 4 vectors
// at n = 40 are 320 CTAs on 152 SMs, three rounds where 2.1 would do; and a
// double-single plane of three fields fills an SM's shared memory, which left
// one CTA per SM, waiting at its own barriers.)
//
// Every pencil is split over G threads, N = G*M (field_split): a whole pencil
// is too much for one thread's registers beyond N ~ 32, and on small grids the
// serial FP64 chain of one thread is what a kernel waits for.  Coprime G, M
// use the prime-factor index map (no twiddle factors):
//   n = (M*n1 + G*n2) mod N,  k = (M*A*k1 + G*B*k2) mod N,
//   A = M^{-1} mod G, B = G^{-1} mod M,
//   X[k] = sum_{n2} W_M^{n2 k2} sum_{n1} x[n] W_G^{n1 k1};
// powers of two the Cooley-Tukey one, n = M*n1 + n2, k = k1 + G*k2, with W_N^{n2 k1}
// between the passes.
// Pass A: the M length-G DFTs over n1 of every pencil, in place in shared
// memory, dealt to the threads in one sequence.  Pass B: thread (k1, pencil)
// takes the length-M DFT over n2 in registers.  The slots are computed at run
// time: the kernels are bound by arithmetic, and branches that make them
// immediate operands diverge in every warp that holds two values of k1 (a
// third more FP64 instructions in pass A at n = 60).
// ---------------------------------------------------------------------------
template <int N> struct Twiddles {
  double c[N], s[N];
};
template <int N> constexpr Twiddles<N> make_twiddles() {
  Twiddles<N> t{};
  for (int i = 0; i < N; ++i) {
    t.c[i] = cs2pi(i, N, 0);
    t.s[i] = cs2pi(i, N, 1);
  }
  return t;
}
// exp(2 pi i m / N), m < N
template <int N> static __constant__ Twiddles<N> kTwiddles = make_twiddles<N>();

FAME_HD constexpr int gcd_of(int a, int b) { return b == 0 ? a : gcd_of(b, a % b); }

template <int N, int G> struct Split {
  static constexpr int M = N / G;
  static constexpr bool PFA = gcd_of(G, M) == 1;
  static constexpr int A = PFA ? fft_inv_mod(M % G, G) : 0;
  static constexpr int B = PFA ? fft_inv_mod(G % M, M) : 0;
  static constexpr int NA = (M + G - 1) / G;          // rounds of pass A
  static_assert(G * M == N, "a split of N");
  FAME_HD static int wrap(int a) { return a >= N ? a - N : a; }
  // element n1 of the DFT n2 of pass A; element n2 of row n1 of pass B
  FAME_HD static int in_slot(int n1, int n2) { return PFA ? wrap(M * n1 + G * n2) : M * n1 + n2; }
  // output k2 of row k1
  FAME_HD static int out_slot(int k1, int k2) {
    return PFA ? wrap((M * A * k1) % N + (G * B * k2) % N) : k1 + G * k2;
  }
};

// One DFT of pass A (S: direction) with the twiddle of the Cooley-Tukey map.
template <class R, int N, int G, int S> __device__ __forceinline__ void pass_a_dft(cx<R> (&a)[G], int n2) {
  fft<R, G, S>(a);
  if constexpr (!Split<N, G>::PFA) {
#pragma unroll
    for (int k1 = 1; k1 < G; ++k1) {
      const double c = kTwiddles<N>.c[n2 * k1], s = kTwiddles<N>.s[n2 * k1];
      a[k1] = cmul(mk<R>(R(c), R(S * s)), a[k1]);
    }
  }
}

// Pass A with T threads on NP pencils; base(p) points at element 0 of pencil
// p, elements STRIDE apart.
template <class R, int N, int G, int S, int STRIDE, int NP, int T, class F>
__device__ __forceinline__ void split_pass_a(int tid, F&& base) {
  using SP = Split<N, G>;
#pragma unroll
  for (int j = 0; j < SP::NA; ++j) {
    const int idx = tid + j * T;
    if (tid < T && idx < NP * SP::M) {
      const int n2 = idx / NP, p = idx - n2 * NP;
      cx<R>* q = base(p);
      cx<R> a[G];
#pragma unroll
      for (int n1 = 0; n1 < G; ++n1) a[n1] = q[SP::in_slot(n1, n2) * STRIDE];
      pass_a_dft<R, N, G, S>(a, n2);
#pragma unroll
      for (int n1 = 0; n1 < G; ++n1) q[SP::in_slot(n1, n2) * STRIDE] = a[n1];
    }
  }
}

// Pass B read: the M values of row k1 of one pencil.
template <class R, int N, int G, int STRIDE>
__device__ __forceinline__ void split_pass_b_load(const cx<R>* p, int k1, cx<R> (&z)[N / G]) {
  using SP = Split<N, G>;
#pragma unroll
  for (int n2 = 0; n2 < SP::M; ++n2) z[n2] = p[SP::in_slot(k1, n2) * STRIDE];
}

// Pass B write: X[out_slot(k1, k2)] = z[k2].
template <class R, int N, int G, int STRIDE>
__device__ __forceinline__ void split_pass_b_store(cx<R>* p, int k1, const cx<R> (&z)[N / G]) {
  using SP = Split<N, G>;
#pragma unroll
  for (int k2 = 0; k2 < SP::M; ++k2) p[SP::out_slot(k1, k2) * STRIDE] = z[k2];
}

template <class R, int N> struct FieldShape {
  static constexpr int G = field_split(N);
  static constexpr int KP = N <= 16 ? 2 : 1;       // planes per CTA: small planes share one, to fill its warps
  static constexpr int NP = KP * N;                // pencils per axis
  static constexpr int T = NP * G;                 // threads of the DFT passes
  static constexpr int TB = ((T + 31) / 32) * 32 < 64 ? 64 : ((T + 31) / 32) * 32;
  // Double-single waits on latencies at two CTAs per SM (n = 60: 128 registers, 36 %
  // issue): up to 24 warps of 80 registers, without spills at the two elements
  // in flight of k_field_inv (ten vectors at n = 60 844 -> 762 us there, one vector's
  // fncB 372 -> 272 as its 360 CTAs then fit at once).  The FP64 rate bounds double.
  static constexpr int CTAS = !std::is_same_v<R, ff> ? 0 : 24 / (TB / 32) > 0 ? 24 / (TB / 32) : 1;
  static constexpr int LD = N + 1;
  static constexpr size_t SMEM = sizeof(cx<R>) * KP * N * LD;
  static_assert(N % KP == 0, "whole CTAs of planes");
};

// Rows of the staged planes (pencil p at sm + p * LD): the length-N DFT along x
// in place; thread (g, p).
template <class R, int N, int S> __device__ __forceinline__ void field_rows(cx<R>* sm, int tid, int g, int p, bool act) {
  using FS = FieldShape<R, N>;
  constexpr int G = FS::G, M = N / G;
  if constexpr (G > 1) {
    split_pass_a<R, N, G, S, 1, FS::NP, FS::T>(tid, [&](int q) { return sm + q * FS::LD; });
    __syncthreads();
  }
  cx<R>* row = sm + p * FS::LD;
  cx<R> z[M];
  if (act) {
    split_pass_b_load<R, N, G, 1>(row, g, z);
    fft<R, M, S>(z);
  }
  if constexpr (G > 1) __syncthreads();
  if (act) split_pass_b_store<R, N, G, 1>(row, g, z);
  __syncthreads();
}

// What a field kernel does with Pi: nothing; the product with it; that and the sum of
// Re(xp^H y) (k_field_fwd); the product with Pi evaluated by the cluster (k_field_inv).
enum { kCopy = 0, kPi = 1, kPiDot = 2, kPiEval = 3 };

// grid: (n / KP, 3 * sides, vectors); blockIdx.y = 3 * (side - side0) + field.
// Double-single takes Pi from the plan's table, its loads all issued before the first
// conversion (8 vectors at n = 40 485 -> 444 us, one at n = 60 268 -> 237), or, for a
// plan that reads no table, evaluates it in clusters (PREP kPiEval): the three
// field CTAs of one (plane, side, vector) each take a third of the voxels, whose two
// square roots and divisions are FP64, and write all three components into each
// other's shared memory.  fncB without the table of 8 vectors at n = 60: 3110 us with
// three fields per CTA, 3500 with each field's CTA evaluating its own component,
// 2660 so.  Complex128, bound by FP64 throughout, tests for the table here
// (4880 us without it; and a kernel for the table alone was slower, n = 12, ten
// vectors 38.3 -> 40.1).
template <class R, int N, int PREP>
__global__ void __launch_bounds__(FieldShape<R, N>::TB, PREP == kPiEval ? 0 : FieldShape<R, N>::CTAS)
k_field_inv(const cx<R>* __restrict__ x, cx<R>* __restrict__ out, PlanData<R> d,
            const __grid_constant__ VecCtx ctx, long long in_stride, long long in_side_stride,
            long long out_stride, int side0) {
  using FS = FieldShape<R, N>;
  constexpr int G = FS::G, M = N / G, LD = FS::LD, KP = FS::KP, TB = FS::TB;
  constexpr int NN = N * N, Nq = NN * N;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cx<R>* sm = reinterpret_cast<cx<R>*>(smem_raw);  // [KP][N][LD]
  const int k3 = blockIdx.x * KP;
  const int vec = blockIdx.z;
  pdl_wait();
  if (ctx.active && !ctx.active[vec]) return;
  const int inst = vec_inst(ctx, vec);
  const int c = blockIdx.y % 3, side = side0 + blockIdx.y / 3;
  const int tid = threadIdx.x;
  const cx<R>* lam = d.lam + (long long)inst * 3 * N;
  const cx<R>* xin = x + vec * in_stride + (blockIdx.y / 3) * in_side_stride + k3 * NN;
  if constexpr (PREP == kPiEval) {
    auto cluster = cooperative_groups::this_cluster();
    cx<R>* f[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) f[k] = cluster.map_shared_rank(sm, k);
    cluster.sync();  // the neighbours run
    for (int e = c * TB + tid; e < KP * NN; e += 3 * TB) {
      const int r = e / N, i1 = e - r * N;
      const cx<R> a = cscale(load_io<R>(xin + e), scale3<R, N>());
      const cx<R> b = cscale(load_io<R>(xin + Nq + e), scale3<R, N>());
      const PiBlock<R> P = pi_block<R>(lam[i1], lam[N + r % N], lam[2 * N + k3 + r / N]);
      // side 1: Pi1 a + Pi2 b; side 0: conj(Pi1) b - conj(Pi2) a (as in k_field_fwd)
      const cx<R> X = side ? a : b, Y = side ? b : cneg(a);
#pragma unroll
      for (int k = 0; k < 3; ++k)
        f[k][r * LD + i1] = cfma(conj_unless(P.p2[k], side), Y, cmul(conj_unless(P.p1[k], side), X));
    }
    cluster.sync();
  } else {
    // the loads of U elements issued together
    constexpr int ITEMS = (KP * NN + TB - 1) / TB;
    constexpr int UMAX = std::is_same_v<R, ff> ? 2 : 4, U = ITEMS < UMAX ? ITEMS : UMAX;
    for (int b = 0; b < ITEMS; b += U) {
      io_t<R> in[U][2];
      PiComp<R> P[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int e = tid + (b + u) * TB;
        if (e < KP * NN) {
          if constexpr (PREP == kPi) {
            in[u][0] = load_raw<R>(xin + e);
            in[u][1] = load_raw<R>(xin + Nq + e);
            if constexpr (std::is_same_v<R, ff>) P[u] = pi_table<R, N>(d, inst, c, k3 * NN + e);
            else P[u] = pi_comp<R, N>(d, inst, c, k3 * NN + e, lam);
          } else {
            in[u][0] = load_raw<R>(xin + (long long)c * Nq + e);
          }
        }
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int e = tid + (b + u) * TB;
        if (e < KP * NN) {
          const int r = e / N, i1 = e - r * N;
          cx<R> v = from_io<R>(in[u][0]);
          if constexpr (PREP == kPi) {
            const cx<R> a = v, b = from_io<R>(in[u][1]);
            if (side == 0) v = cfmac(P[u].p1, b, cneg(cmulc(P[u].p2, a)));
            else v = cfma(P[u].p2, b, cmul(P[u].p1, a));
          }
          sm[r * LD + i1] = v;
        }
      }
    }
    __syncthreads();
  }
  const int g = tid / FS::NP, p = tid - g * FS::NP;
  const bool act = tid < FS::T;
  field_rows<R, N, +1>(sm, tid, g, p, act);
  // y columns, written straight to global
  auto column = [&](int q) { return sm + (q / N) * N * LD + q % N; };
  if constexpr (G > 1) {
    split_pass_a<R, N, G, +1, LD, FS::NP, FS::T>(tid, column);
    __syncthreads();
  }
  if (act) {
    cx<R> z[M];
    split_pass_b_load<R, N, G, LD>(column(p), g, z);
    fft<R, M, +1>(z);
    cx<R>* o = out + vec * out_stride + (long long)blockIdx.y * Nq + (k3 + p / N) * NN + p % N;
    split_pass_b_store<R, N, G, N>(o, g, z);
  }
}

// POST: the three field CTAs of one (plane, side, vector) form a cluster; each
// applies Pi^H on a third of the voxels, reading the other two fields from
// its neighbours' shared memory.  POST 2 also sums Re(xp^H y) over the CTA's
// voxels for xp laid out as y (one partial per CTA): in a CG iteration one
// pass over p and q less (c128, two vectors at n = 30: a launch of 5.3 us).
template <class R, int N, int POST>
__global__ void __launch_bounds__(FieldShape<R, N>::TB, FieldShape<R, N>::CTAS)
k_field_fwd(const cx<R>* __restrict__ w, cx<R>* __restrict__ y, PlanData<R> d,
            const __grid_constant__ VecCtx ctx, long long w_stride, long long out_stride,
            long long out_side_stride, int side0, const cx<R>* __restrict__ xp, double2* __restrict__ pq) {
  using FS = FieldShape<R, N>;
  constexpr int G = FS::G, M = N / G, LD = FS::LD, KP = FS::KP, TB = FS::TB;
  constexpr int NN = N * N, Nq = NN * N;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cx<R>* sm = reinterpret_cast<cx<R>*>(smem_raw);  // [KP][N][LD]
  const int k3 = blockIdx.x * KP;
  const int vec = blockIdx.z;
  pdl_wait();
  if (ctx.active && !ctx.active[vec]) return;  // the same for a whole cluster
  const int inst = vec_inst(ctx, vec);
  const int c = blockIdx.y % 3, side = side0 + blockIdx.y / 3;
  const int tid = threadIdx.x;
  const int g = tid / FS::NP, p = tid - g * FS::NP;
  const bool act = tid < FS::T;
  // y columns, pass A (G = 1: the whole DFT) straight from global, every load
  // of a thread issued before the first is used
  const cx<R>* src = w + vec * w_stride + (long long)blockIdx.y * Nq + k3 * NN;
  auto column = [&](int q) { return sm + (q / N) * N * LD + q % N; };
  if constexpr (G > 1) {
    using SP = Split<N, G>;
    cx<R> a[SP::NA][G];
#pragma unroll
    for (int j = 0; j < SP::NA; ++j) {
      const int idx = tid + j * FS::T;
      if (act && idx < FS::NP * M) {
        const int n2 = idx / FS::NP, q = idx - n2 * FS::NP;
#pragma unroll
        for (int n1 = 0; n1 < G; ++n1) a[j][n1] = src[(q / N) * NN + SP::in_slot(n1, n2) * N + q % N];
      }
    }
#pragma unroll
    for (int j = 0; j < SP::NA; ++j) {
      const int idx = tid + j * FS::T;
      if (act && idx < FS::NP * M) {
        const int n2 = idx / FS::NP;
        cx<R>* col = column(idx - n2 * FS::NP);
        pass_a_dft<R, N, G, -1>(a[j], n2);
#pragma unroll
        for (int n1 = 0; n1 < G; ++n1) col[SP::in_slot(n1, n2) * LD] = a[j][n1];
      }
    }
    __syncthreads();
    cx<R> z[M];
    if (act) {
      split_pass_b_load<R, N, G, LD>(column(p), g, z);
      fft<R, M, -1>(z);
    }
    __syncthreads();
    if (act) split_pass_b_store<R, N, G, LD>(column(p), g, z);
  } else if (act) {
    cx<R> v[N];
#pragma unroll
    for (int i2 = 0; i2 < N; ++i2) v[i2] = src[(p / N) * NN + i2 * N + p % N];
    fft<R, N, -1>(v);
    cx<R>* col = column(p);
#pragma unroll
    for (int i2 = 0; i2 < N; ++i2) col[i2 * LD] = v[i2];
  }
  __syncthreads();
  field_rows<R, N, -1>(sm, tid, g, p, act);
  const long long oo = vec * out_stride + (blockIdx.y / 3) * out_side_stride + k3 * NN;
  cx<R>* o = y + oo;
  if constexpr (POST != kCopy) {
    double dot = 0.0;
    auto cluster = cooperative_groups::this_cluster();
    cluster.sync();
    const cx<R>* u0 = cluster.map_shared_rank(sm, 0);
    const cx<R>* u1 = cluster.map_shared_rank(sm, 1);
    const cx<R>* u2 = cluster.map_shared_rank(sm, 2);
    const cx<R>* lam = d.lam + (long long)inst * 3 * N;
    for (int e = c * TB + tid; e < KP * NN; e += 3 * TB) {
      const int r = e / N, i1 = e - r * N;
      const int q = r * LD + i1;
      cx<R> xa, xb;
      if constexpr (POST == kPiDot) {
        xa = xp[oo + e];
        xb = xp[oo + Nq + e];
      }
      const cx<R> f[3] = {u0[q], u1[q], u2[q]};
      // side 1: a = X, b = Y with X = sum conj(Pi1) v, Y = sum conj(Pi2) v;
      // side 0: a = -Y, b = X with conj(Pi) for Pi (one instruction stream:
      // two branches are computed both and selected)
      cx<R> X, Y;
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        const PiComp<R> P = pi_comp<R, N>(d, inst, k, k3 * NN + e, lam);
        const cx<R> p1 = conj_unless(P.p1, side), p2 = conj_unless(P.p2, side);
        X = k == 0 ? cmulc(p1, f[k]) : cfmac(p1, f[k], X);
        Y = k == 0 ? cmulc(p2, f[k]) : cfmac(p2, f[k], Y);
      }
      const cx<R> a = side ? X : cneg(Y), b = side ? Y : X;
      store_io<R>(o + e, a);
      store_io<R>(o + Nq + e, b);
      if constexpr (POST == kPiDot)
        dot = rfma(xa.x, a.x, rfma(xa.y, a.y, rfma(xb.x, b.x, rfma(xb.y, b.y, dot))));
    }
    if constexpr (POST == kPiDot) {
      __shared__ double sh[TB];
      sh[tid] = dot;
      cluster.sync();
      if (tid < 32) {
#pragma unroll
        for (int k = 1; k < TB / 32; ++k) dot += sh[tid + 32 * k];
#pragma unroll
        for (int k = 16; k > 0; k >>= 1) dot += __shfl_down_sync(0xffffffffu, dot, k);
        if (tid == 0)
          pq[(long long)vec * gridDim.x * gridDim.y + blockIdx.y * gridDim.x + blockIdx.x] = make_double2(dot, 0.0);
      }
    } else {
      cluster.sync();  // no CTA leaves while its shared memory is read
    }
  } else {
    for (int e = tid; e < KP * NN; e += TB) {
      const int r = e / N, i1 = e - r * N;
      o[(long long)c * Nq + e] = sm[r * LD + i1];
    }
  }
}

// ---------------------------------------------------------------------------
// col: DFT along z of every (i1, i2) column, src -> dst (which may be the
// same).  SMODE 1: multiply the Bloch phase S = S_x S_y S_z and scale after
// (inverse); 2: conj(S) and scale before (forward); 0: neither.
//
// complex64: k_col, one thread per column (N complex values in registers,
// loads and stores coalesced along x).
// ---------------------------------------------------------------------------
template <int N, int DIR, int SMODE>
__global__ void __launch_bounds__(128, 3)
k_col(const float2* src, float2* dst, PlanData<float> d, const __grid_constant__ VecCtx ctx,
      long long stride, float scale) {
  const int col = blockIdx.x * blockDim.x + threadIdx.x;
  const int f = blockIdx.y;
  const int vec = blockIdx.z;
  pdl_wait();
  if (col >= N * N) return;
  if (ctx.active && !ctx.active[vec]) return;
  const long long Nq = (long long)N * N * N;
  const long long off = vec * stride + (long long)f * Nq + col;
  const float2* p = src + off;
  float2* o = dst + off;
  const float2* S = d.sxyz + (long long)vec_inst(ctx, vec) * 3 * N;
  float2 sxy = zero<float>();
  if constexpr (SMODE != 0) sxy = cscale(cmul(S[col % N], S[N + col / N]), scale);
  float2 v[N];
#pragma unroll
  for (int i = 0; i < N; ++i) {
    v[i] = p[(long long)i * N * N];
    if constexpr (SMODE == 2) v[i] = cmulc(cmul(S[2 * N + i], sxy), v[i]);
  }
  fft<float, N, DIR>(v);
#pragma unroll
  for (int i = 0; i < N; ++i) {
    float2 r = v[i];
    if constexpr (SMODE == 1) r = cmul(cmul(S[2 * N + i], sxy), r);
    o[(long long)i * N * N] = r;
  }
}

// complex128 and double-single: k_col2, with the split of the field kernels.
// One CTA per (W columns, field, vector), W*G threads: pass A straight from
// global, pass B straight to global.  With W = 32 a warp holds one k1 of 32
// columns (no idle lanes: whole rows of 40 columns took 52 us where this takes
// 44, 4 vectors at n = 40); an even split takes 16, two k1 to a warp, as smaller
// CTAs leave the SMs more evenly loaded (615 of 32 columns for five transforms at
// n = 36 put 5 on some SMs and 4 on the others: 89 us, 83 with 16; fncB of one
// vector at n = 32 81 -> 78, at n = 50 313 -> 305).  (One thread per 60-point column needs 255
// registers and spills; at n = 16 it is a serial chain of 170 FP64 operations.)
template <int N> FAME_HD constexpr int col_width() { return N <= 16 || field_split(N) % 2 == 0 ? 16 : 32; }

template <class R, int N, int DIR, int SMODE>
__global__ void __launch_bounds__(((col_width<N>() * field_split(N) + 31) / 32) * 32)
k_col2(const cx<R>* src, cx<R>* dst, PlanData<R> d, const __grid_constant__ VecCtx ctx, long long stride, R scale) {
  constexpr int G = field_split(N);
  using SP = Split<N, G>;
  constexpr int M = SP::M, W = col_width<N>(), LD = W + 1, T = W * G, NN = N * N;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cx<R>* sm = reinterpret_cast<cx<R>*>(smem_raw);  // [z][LD]
  const int vec = blockIdx.z;
  pdl_wait();
  if (ctx.active && !ctx.active[vec]) return;
  const int tid = threadIdx.x;
  const int g = tid / W, x = tid - g * W;  // T threads: row k1 = g of column col
  const int col = blockIdx.x * W + x;
  const bool act = tid < T && col < NN;
  const long long off = vec * stride + (long long)blockIdx.y * N * NN + blockIdx.x * W;
  const cx<R>* p = src + off;
  cx<R>* o = dst + off;
  const cx<R>* S = d.sxyz + (long long)vec_inst(ctx, vec) * 3 * N;
  cx<R> sxy = zero<R>();
  if constexpr (SMODE != 0) sxy = cscale(cmul(S[col % N], S[N + (col / N) % N]), scale);
  if constexpr (G > 1) {
    cx<R> a[SP::NA][G];
#pragma unroll
    for (int j = 0; j < SP::NA; ++j) {
      const int n2 = g + j * G;  // the round's DFTs n2 of this column
      if (act && n2 < M) {
#pragma unroll
        for (int n1 = 0; n1 < G; ++n1) {
          const int z = SP::in_slot(n1, n2);
          a[j][n1] = p[z * NN + x];
          if constexpr (SMODE == 2) a[j][n1] = cmulc(cmul(S[2 * N + z], sxy), a[j][n1]);
        }
      }
    }
#pragma unroll
    for (int j = 0; j < SP::NA; ++j) {
      const int n2 = g + j * G;
      if (act && n2 < M) {
        pass_a_dft<R, N, G, DIR>(a[j], n2);
#pragma unroll
        for (int n1 = 0; n1 < G; ++n1) sm[SP::in_slot(n1, n2) * LD + x] = a[j][n1];
      }
    }
    __syncthreads();
  }
  if (act) {
    cx<R> z[M];
    if constexpr (G > 1) {
      split_pass_b_load<R, N, G, LD>(sm + x, g, z);
    } else {
#pragma unroll
      for (int i = 0; i < M; ++i) {
        z[i] = p[i * NN + x];
        if constexpr (SMODE == 2) z[i] = cmulc(cmul(S[2 * N + i], sxy), z[i]);
      }
    }
    fft<R, M, DIR>(z);
#pragma unroll
    for (int k2 = 0; k2 < M; ++k2) {
      const int k = SP::out_slot(g, k2);
      cx<R> r = z[k2];
      if constexpr (SMODE == 1) r = cmul(cmul(S[2 * N + k], sxy), r);
      o[k * NN + x] = r;
    }
  }
}

template <class R, int N, bool PREP>
cudaError_t plane_inv(const PlanData<R>& d, const cx<R>* x, cx<R>* out, int nvec, int nside, int side0,
                      long long in_stride, long long in_side_stride, long long out_stride, const VecCtx& ctx,
                      cudaStream_t st) {
  if constexpr (sizeof(cx<R>) == 8) {
    return launch<k_plane_inv<N, PREP>>(dim3(N, nside, nvec), ((3 * N + 31) / 32) * 32, plane_smem<N>(), st, x, out,
                                            d, ctx, in_stride, in_side_stride, out_stride, side0);
  } else {
    using FS = FieldShape<R, N>;
    const dim3 g(N / FS::KP, 3 * nside, nvec);
    if constexpr (PREP && std::is_same_v<R, ff>)
      if (!d.pi)
        return launch<k_field_inv<R, N, kPiEval>, 3>(g, FS::TB, FS::SMEM, st, x, out, d, ctx, in_stride, in_side_stride,
                                                     out_stride, side0);
    return launch<k_field_inv<R, N, PREP ? kPi : kCopy>>(g, FS::TB, FS::SMEM, st, x, out, d, ctx, in_stride,
                                                         in_side_stride, out_stride, side0);
  }
}

template <class R, int N, bool POST>
cudaError_t plane_fwd(const PlanData<R>& d, const cx<R>* w, cx<R>* y, int nvec, int nside, int side0,
                      long long w_stride, long long out_stride, long long out_side_stride, const VecCtx& ctx,
                      cudaStream_t st, const cx<R>* xp = nullptr, double2* pq = nullptr) {
  if constexpr (sizeof(cx<R>) == 8) {
    return launch<k_plane_fwd<N, POST>>(dim3(N, nside, nvec), ((3 * N + 31) / 32) * 32, plane_smem<N>(), st, w, y, d,
                                            ctx, w_stride, out_stride, out_side_stride, side0);
  } else {
    using FS = FieldShape<R, N>;
    const dim3 g(N / FS::KP, 3 * nside, nvec);
    if constexpr (POST && std::is_same_v<R, double>)
      if (pq)
        return launch<k_field_fwd<R, N, kPiDot>, 3>(g, FS::TB, FS::SMEM, st, w, y, d, ctx, w_stride, out_stride,
                                                    out_side_stride, side0, xp, pq);
    return launch<k_field_fwd<R, N, POST ? kPi : kCopy>, POST ? 3 : 1>(g, FS::TB, FS::SMEM, st, w, y, d, ctx, w_stride,
                                                                       out_stride, out_side_stride, side0, xp, pq);
  }
}

template <class R, int N, int DIR, int SMODE>
cudaError_t col(const Plan& P, const PlanData<R>& d, const cx<R>* src, cx<R>* dst, int nfield, int nvec,
                long long stride, const VecCtx& ctx, cudaStream_t st, R scale = R(1)) {
  if constexpr (sizeof(cx<R>) == 16) {
    constexpr int G = field_split(N), W = col_width<N>();
    return launch<k_col2<R, N, DIR, SMODE>>(dim3((N * N + W - 1) / W, nfield, nvec), ((W * G + 31) / 32) * 32,
                                                G > 1 ? sizeof(cx<R>) * N * (W + 1) : 0, st, src, dst, d, ctx, stride,
                                                scale);
  } else {
    // one warp per CTA for small batches, so that the work spreads over the
    // SMs, 128 threads where there are plenty
    const int tpb = (long long)N * N * nfield * nvec < 128LL * 6 * P.sms ? 32 : 128;
    return launch<k_col<N, DIR, SMODE>>(dim3((N * N + tpb - 1) / tpb, nfield, nvec), tpb, 0, st, src, dst, d, ctx,
                                            stride, scale);
  }
}


// fncB on a batch, as sub-batches of `chunk` vectors (0: all at once) so that
// the six-field intermediates of a sub-batch can stay in L2; the stencil
// kernels run with tpb threads per block.  Both come from fame_autotune.
//
// pq (may be null): per-CTA partial sums of Re(x^H B x), pq_partials_n per vector,
// vector-major.  With the single-pass stencil: the curl-SVD transforms are
// unitary and Pi has orthonormal columns, so x^H B x equals w^H [M J^H; J N] w for
// the spatial fields w the stencil reads; the stencil pass accumulates it while
// it writes its output.  With the two-kernel form of complex128: the last kernel
// does, from x and the y it writes.
template <class R, int N> int pq_partials_n(const Plan& P, const TuneEntry& tn, int nvec) {
  if (tn.stencil_tpb == 0) return sweep_partials_n<R, N>(sweep_planes<R, N>(P, sub_batch(tn, nvec)));
  return std::is_same_v<R, double> ? 6 * N / FieldShape<R, N>::KP : 0;
}
template <class R, int N>
cudaError_t fncB_n(const Plan& P, const cx<R>* x, cx<R>* y, int nvec, const VecCtx& ctx, cx<R>* w0, cx<R>* w1,
                   cudaStream_t st, double2* pq) {
  PlanData<R> d = pdata<R>(P);
  if (!P.opt_pi_table) d.pi = nullptr;  // evaluate Pi in the plane kernels instead
  const long long Nq = P.Nq;
  const TuneEntry tn = tune_for(P, tune_prec<R>(), nvec);
  const int chunk = sub_batch(tn, nvec);
  const int tz = sweep_planes<R, N>(P, chunk), npq = pq_partials_n<R, N>(P, tn, nvec);
  for (int v0 = 0; v0 < nvec; v0 += chunk) {
    const int nv = std::min(chunk, nvec - v0);
    const VecCtx c = sub_ctx(ctx, v0);
    const cx<R>* xs = x + (size_t)v0 * 4 * Nq;
    cx<R>* ys = y + (size_t)v0 * 4 * Nq;
    cudaError_t e;
    e = plane_inv<R, N, true>(d, xs, w0, nv, 2, 0, 4 * Nq, 2 * Nq, 6 * Nq, c, st);
    if (e != cudaSuccess) return e;
    e = col<R, N, +1, 0>(P, d, w0, w0, 6, nv, 6 * Nq, c, st);
    if (e != cudaSuccess) return e;
    double2* pqs = pq ? pq + (size_t)v0 * npq : nullptr;
    // material stencil: single pass w0 -> w1, or the two-kernel form in place on w0
    cx<R>* wm = w0;
    if (tn.stencil_tpb == 0) {
      e = sweep_n<R, N>(P, w0, w1, nv, c, st, tz, pqs);
      wm = w1;
    } else {
      e = stencil_n<R, N>(P, w0, w0, w1, nv, c, st, tn.stencil_tpb, false);
    }
    if (e != cudaSuccess) return e;
    e = col<R, N, -1, 0>(P, d, wm, wm, 6, nv, 6 * Nq, c, st);
    if (e != cudaSuccess) return e;
    e = plane_fwd<R, N, true>(d, wm, ys, nv, 2, 0, 6 * Nq, 4 * Nq, 2 * Nq, c, st, xs,
                              tn.stencil_tpb == 0 ? nullptr : pqs);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

template <class R, int N>
cudaError_t fields_inv_n(const Plan& P, const cx<R>* x, cx<R>* w, int nvec, const VecCtx& ctx, cudaStream_t st) {
  const PlanData<R>& d = pdata<R>(P);
  const long long Nq = P.Nq;
  cudaError_t e = plane_inv<R, N, true>(d, x, w, nvec, 2, 0, 4 * Nq, 2 * Nq, 6 * Nq, ctx, st);
  if (e != cudaSuccess) return e;
  return col<R, N, +1, 0>(P, d, w, w, 6, nvec, 6 * Nq, ctx, st);
}

template <class R, int N>
cudaError_t transform_n(const Plan& P, int trans, const cx<R>* x, cx<R>* y, int nvec, const VecCtx& ctx,
                        cudaStream_t st) {
  const PlanData<R>& d = pdata<R>(P);
  const long long Nq = P.Nq;
  const R scale = R(1.0 / (double(N) * csqrt_int(N)));
  cudaError_t e;
  if (trans == 0) {
    e = plane_inv<R, N, false>(d, x, y, nvec, 1, 0, 3 * Nq, 0, 3 * Nq, ctx, st);
    if (e != cudaSuccess) return e;
    return col<R, N, +1, 1>(P, d, y, y, 3, nvec, 3 * Nq, ctx, st, scale);
  }
  // transpose: z first (with conj(S) before), then y, x
  e = col<R, N, -1, 2>(P, d, x, y, 3, nvec, 3 * Nq, ctx, st, scale);
  if (e != cudaSuccess) return e;
  return plane_fwd<R, N, false>(d, y, y, nvec, 1, 0, 3 * Nq, 3 * Nq, 0, ctx, st);
}

template <class R, int N>
cudaError_t handle_n(const Plan& P, int which, const cx<R>* x, cx<R>* y, int nvec, const VecCtx& ctx,
                     cx<R>* w0, cudaStream_t st) {
  const PlanData<R>& d = pdata<R>(P);
  const long long Nq = P.Nq;
  cudaError_t e;
  if (which == 0 || which == 1) {  // Pr / Qr : 2Nq -> 3Nq
    e = plane_inv<R, N, true>(d, x, y, nvec, 1, which, 2 * Nq, 0, 3 * Nq, ctx, st);
    if (e != cudaSuccess) return e;
    return col<R, N, +1, 1>(P, d, y, y, 3, nvec, 3 * Nq, ctx, st);
  }
  // Prs / Qrs : 3Nq -> 2Nq through the 3Nq scratch w0
  e = col<R, N, -1, 2>(P, d, x, w0, 3, nvec, 3 * Nq, ctx, st);
  if (e != cudaSuccess) return e;
  return plane_fwd<R, N, true>(d, w0, y, nvec, 1, which - 2, 3 * Nq, 2 * Nq, 0, ctx, st);
}


}  // namespace detail
}  // namespace fame

// Declarations of the size-templated entry points of one (precision, size),
// each prefixed by PFX ("template" to instantiate, "extern template" to
// suppress instantiation in other translation units).
#define FAME_SIZE_SIGS(PFX, R, NN)                                                                                 \
  PFX cudaError_t fame::detail::fncB_n<R, NN>(const Plan&, const cx<R>*, cx<R>*, int, const VecCtx&, cx<R>*,       \
                                              cx<R>*, cudaStream_t, double2*);                                    \
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
// The grid sizes of the band solves that it was written for.  fncB of one and of eight
// vectors, double-single against FP64 (us): n = 12 30 33 / 29 34, 24 46 103 / 47 176,
// 40 78 443 / 128 802, 48 131 838 / 203 1412, 60 242 1640 / 408 2721.  The kernels compile for
// every size, and measured so it would gain at most of the others too: n = 16 34 48 / 31 60,
// 18 50 68 / 45 102, 20 40 69 / 36 110, 30 70 224 / 77 340, 32 60 241 / 78 414, 36 74 355 /
// 111 618, 50 345 1863 / 307 2007, 64 309 2021 / 516 3733; all of them together take the
// build from 38 to 53 s.
#define FAME_FOR_EACH_DS_N(X) X(12) X(24) X(40) X(48) X(60)
#define FAME_DS_SIGS(PFX, NN)                                                                                      \
  PFX cudaError_t fame::detail::fncB_n<fame::ff, NN>(const Plan&, const cx<fame::ff>*, cx<fame::ff>*, int,         \
                                                     const VecCtx&, cx<fame::ff>*, cx<fame::ff>*, cudaStream_t,    \
                                                     double2*);
#define FAME_INST_DS(NN) FAME_DS_SIGS(template, NN)

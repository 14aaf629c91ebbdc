// Material stencil of fncB on the six spatial fields.
//
// Two forms:
//   k_sweep             : one pass, the fields read once (out of place);
//   k_vertex, k_faceedge: U, V gathered to every vertex and Hu, Hv = vertex
//                         tensor products into scratch h, then u', v' from
//                         the fields and h.  One thread per voxel.
// Size templated (instantiated per grid size with the transforms in
// fncb_inst_*.cu) so that the index arithmetic is 32-bit with compile-time
// divisors.
//
// The factors 1/4, 1/2 of the gathers and scatters are folded into the vertex
// tensors (powers of two: exact), which the plan keeps in the order the
// kernels read them, per instance and phase (PlanData::stn):
//   general (36 reals): D0..5 | M01 M02 M12 | N01 N02 N12 | J (row-major, complex)
//   chiral  (24 reals): D0..5 | M01 M02 M12 | N01 N02 N12 | Im J (9) | 3 unused
// with D = (Re Mh_ii / 4, Re Nh_ii / 2), M = Mh_ij / 16, N = Nh_ij / 4, J / 8.
// "Chiral" means every phase of every instance has real N and M and imaginary
// J, exactly: the bi-isotropic media eps, mu, xi = -zeta = i gamma of the
// crystals here (a real lattice congruence keeps the property).  Skipping the
// zero halves takes the vertex product from 120 to 60 multiply-adds.
#pragma once

#include "fame_internal.h"
#include "launch.h"

namespace fame {
namespace detail {

template <class R> inline const PlanData<R>& pdata(const Plan& P);
template <> inline const PlanData<double>& pdata<double>(const Plan& P) { return P.d64; }
template <> inline const PlanData<float>& pdata<float>(const Plan& P) { return P.d32; }
template <> inline const PlanData<ff>& pdata<ff>(const Plan& P) { return P.dds; }

// The CNT reals of one stored vertex tensor (16-byte loads where R is float).
template <class R, int CNT> __device__ __forceinline__ void load_tensor(const R* p, R (&t)[CNT]) {
  if constexpr (sizeof(R) == 4) {
    const float4* q = reinterpret_cast<const float4*>(p);
#pragma unroll
    for (int i = 0; i < CNT / 4; ++i) {
      const float4 v = q[i];
      t[4 * i] = v.x;
      t[4 * i + 1] = v.y;
      t[4 * i + 2] = v.z;
      t[4 * i + 3] = v.w;
    }
  } else {
#pragma unroll
    for (int i = 0; i < CNT; ++i) t[i] = p[i];
  }
}

// Vertex product (all scale factors in the tensors): hu, hv and the real
// diagonals dg of one vertex.  KIND: kMatGeneral / kMatChiral from the table
// entry `tab`, kMatField from the fields a | b | g at fld[0], [Nq], [2 Nq].
//   Hu_i = sum_{j!=i} Mh_ij U_j + sum_j conj(J_ji) V_j
//   Hv_i = sum_{j!=i} Nh_ij V_j + sum_j J_ij U_j
template <class R, int KIND>
__device__ __forceinline__ void vertex_product(const R* tab, const R* fld, int Nq, const R* gram, const cx<R> (&U)[3],
                                               const cx<R> (&V)[3], cx<R> (&hu)[3], cx<R> (&hv)[3], R (&dg)[6]) {
  if constexpr (KIND == kMatField) {  // Mh = b G, Nh = a G, J = -i g G
    const R a = fld[0], b = fld[Nq], g = fld[2 * Nq] * R(0.125);
    const R a4 = a * R(0.25), b16 = b * R(0.0625);
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      cx<R> su = zero<R>(), sv = zero<R>();
#pragma unroll
      for (int j = 0; j < 3; ++j)
        if (j != i) {
          su = caxpy(gram[i * 3 + j], U[j], su);
          sv = caxpy(gram[i * 3 + j], V[j], sv);
        }
      const cx<R> tu = caxpy(gram[i * 4], U[i], su), tv = caxpy(gram[i * 4], V[i], sv);
      hu[i] = caxpyi(g, tv, cscale(su, b16));
      hv[i] = caxpyi(-g, tu, cscale(sv, a4));
      dg[i] = b * gram[i * 4] * R(0.25);
      dg[3 + i] = a * gram[i * 4] * R(0.5);
    }
  } else if constexpr (KIND == kMatChiral) {
    R t[kStnChiral];
    load_tensor<R, kStnChiral>(tab, t);
    auto three = [&](const R* o, const cx<R> (&W)[3], cx<R> (&h)[3]) {  // real symmetric, zero diagonal
      h[0] = caxpy(o[0], W[1], cscale(W[2], o[1]));
      h[1] = caxpy(o[0], W[0], cscale(W[2], o[2]));
      h[2] = caxpy(o[1], W[0], cscale(W[1], o[2]));
    };
    three(t + 6, U, hu);
    three(t + 9, V, hv);
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        hu[i] = caxpyi(-t[12 + j * 3 + i], V[j], hu[i]);
        hv[i] = caxpyi(t[12 + i * 3 + j], U[j], hv[i]);
      }
#pragma unroll
    for (int i = 0; i < 6; ++i) dg[i] = t[i];
  } else {
    R t[kStnGeneral];
    load_tensor<R, kStnGeneral>(tab, t);
    auto c = [&](int i) { return mk<R>(t[i], t[i + 1]); };
    auto three = [&](int o, const cx<R> (&W)[3], cx<R> (&h)[3]) {  // Hermitian, zero diagonal
      const cx<R> m01 = c(o), m02 = c(o + 2), m12 = c(o + 4);
      h[0] = cfma(m01, W[1], cmul(m02, W[2]));
      h[1] = cfmac(m01, W[0], cmul(m12, W[2]));
      h[2] = cfmac(m02, W[0], cmulc(m12, W[1]));
    };
    three(6, U, hu);
    three(12, V, hv);
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        hu[i] = cfmac(c(18 + 2 * (j * 3 + i)), V[j], hu[i]);
        hv[i] = cfma(c(18 + 2 * (i * 3 + j)), U[j], hv[i]);
      }
#pragma unroll
    for (int i = 0; i < 6; ++i) dg[i] = t[i];
  }
}

// Shift phases of one voxel for the two-kernel form: T_d of the step to the
// neighbour r + e_d (up) or r - e_d (the conjugate is applied).  Periodic
// frame: tau_d everywhere; Bloch frame: exp(i theta_d) where the step wraps,
// 1 elsewhere.
template <class R, int N>
__device__ __forceinline__ void shift_phases(const PlanData<R>& d, int inst, bool bloch, bool wx, bool wy, bool wz,
                                             cx<R> (&t)[3]) {
#pragma unroll
  for (int a = 0; a < 3; ++a) t[a] = d.tau[inst * 3 + a];
  if (bloch) {
    const bool w[3] = {wx, wy, wz};
#pragma unroll
    for (int a = 0; a < 3; ++a)
      t[a] = w[a] ? cmul(d.sxyz[(inst * 3 + a) * N + N - 1], t[a]) : mk<R>(R(1), R(0));
  }
}

template <class R, int N, int KIND>
__global__ void __launch_bounds__(512)
k_vertex(const cx<R>* __restrict__ uv, cx<R>* __restrict__ h, PlanData<R> d,
         const uint8_t* __restrict__ phase, int nphase, const __grid_constant__ VecCtx ctx, long long stride,
         bool bloch) {
  constexpr int NN = N * N, Nq = NN * N;
  const int idx = blockIdx.x * blockDim.x + threadIdx.x;
  const int vec = blockIdx.y;
  pdl_wait();
  if (idx >= Nq) return;
  if (ctx.active && !ctx.active[vec]) return;
  const int inst = vec_inst(ctx, vec);
  const int i1 = idx % N, i2 = (idx / N) % N, i3 = idx / NN;
  const int dxm = i1 == 0 ? N - 1 : -1;
  const int dym = i2 == 0 ? (N - 1) * N : -N;
  const int dzm = i3 == 0 ? (N - 1) * NN : -NN;
  cx<R> T[3];
  shift_phases<R, N>(d, inst, bloch, i1 == 0, i2 == 0, i3 == 0, T);
  const cx<R>* f = uv + vec * stride + idx;
  // (I + T_a^H)(I + T_b^H) u_j ; (T^H g)(r) = conj(T) g(r - e)
  auto face2vtx = [&](const cx<R>* g, int da, int db, cx<R> ta, cx<R> tb) {
    const cx<R> s0 = cfmac(tb, g[db], g[0]);
    const cx<R> s1 = cfmac(tb, g[da + db], g[da]);
    return cfmac(ta, s1, s0);
  };
  cx<R> U[3], V[3];
  U[0] = face2vtx(f, dym, dzm, T[1], T[2]);
  U[1] = face2vtx(f + Nq, dxm, dzm, T[0], T[2]);
  U[2] = face2vtx(f + 2 * Nq, dxm, dym, T[0], T[1]);
  V[0] = cfmac(T[0], f[3 * Nq + dxm], f[3 * Nq]);
  V[1] = cfmac(T[1], f[4 * Nq + dym], f[4 * Nq]);
  V[2] = cfmac(T[2], f[5 * Nq + dzm], f[5 * Nq]);
  cx<R>* o = h + vec * stride + idx;
  cx<R> hu[3], hv[3];
  R dg[6];
  const R* tab = KIND == kMatField ? nullptr : d.stn + (size_t)(inst * nphase + __ldg(phase + idx)) * stn_size(KIND);
  vertex_product<R, KIND>(tab, d.fld + idx, Nq, d.gram, U, V, hu, hv, dg);
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    o[i * Nq] = hu[i];
    o[(3 + i) * Nq] = hv[i];
  }
}

template <class R, int N, int KIND>
__global__ void __launch_bounds__(512)
k_faceedge(const cx<R>* uv, const cx<R>* __restrict__ h, cx<R>* out, PlanData<R> d,
           const uint8_t* __restrict__ phase, int nphase, const __grid_constant__ VecCtx ctx, long long stride,
           bool bloch) {
  constexpr int NN = N * N, Nq = NN * N;
  const int idx = blockIdx.x * blockDim.x + threadIdx.x;
  const int vec = blockIdx.y;
  pdl_wait();
  if (idx >= Nq) return;
  if (ctx.active && !ctx.active[vec]) return;
  const int inst = vec_inst(ctx, vec);
  const int i1 = idx % N, i2 = (idx / N) % N, i3 = idx / NN;
  const int dxp = i1 == N - 1 ? -(N - 1) : 1;
  const int dyp = i2 == N - 1 ? -(N - 1) * N : N;
  const int dzp = i3 == N - 1 ? -(N - 1) * NN : NN;
  cx<R> T[3];
  shift_phases<R, N>(d, inst, bloch, i1 == N - 1, i2 == N - 1, i3 == N - 1, T);
  // material diagonals at the corners r + {0,1}^3
  R m0, m1, m2, n0, n1, n2;
  if constexpr (KIND == kMatField) {  // Re Mh_ii = b G_ii, Re Nh_ii = a G_ii
    const R* fa = d.fld + idx;
    const R* fb = d.fld + Nq + idx;
    m0 = R(0.25) * d.gram[0] * (fb[0] + fb[dyp] + fb[dzp] + fb[dyp + dzp]);
    m1 = R(0.25) * d.gram[4] * (fb[0] + fb[dxp] + fb[dzp] + fb[dxp + dzp]);
    m2 = R(0.25) * d.gram[8] * (fb[0] + fb[dxp] + fb[dyp] + fb[dxp + dyp]);
    n0 = R(0.5) * d.gram[0] * (fa[0] + fa[dxp]);
    n1 = R(0.5) * d.gram[4] * (fa[0] + fa[dyp]);
    n2 = R(0.5) * d.gram[8] * (fa[0] + fa[dzp]);
  } else {
    const R* tab = d.stn + (size_t)inst * nphase * stn_size(KIND);
    const uint8_t* ph = phase + idx;
    const int p000 = __ldg(ph), p100 = __ldg(ph + dxp), p010 = __ldg(ph + dyp), p001 = __ldg(ph + dzp);
    const int p110 = __ldg(ph + dxp + dyp), p101 = __ldg(ph + dxp + dzp), p011 = __ldg(ph + dyp + dzp);
    auto D = [&](int p, int i) { return tab[p * stn_size(KIND) + i]; };
    m0 = D(p000, 0) + D(p010, 0) + D(p001, 0) + D(p011, 0);
    m1 = D(p000, 1) + D(p100, 1) + D(p001, 1) + D(p101, 1);
    m2 = D(p000, 2) + D(p100, 2) + D(p010, 2) + D(p110, 2);
    n0 = D(p000, 3) + D(p100, 3);
    n1 = D(p000, 4) + D(p010, 4);
    n2 = D(p000, 5) + D(p001, 5);
  }
  const cx<R>* hh = h + vec * stride + idx;
  const cx<R>* f = uv + vec * stride + idx;
  // u'_i = m_i u_i + (I+T_a)(I+T_b) Hu_i ; (T g)(r) = T g(r + e)
  auto vtx2face = [&](const cx<R>* g, int da, int db, cx<R> ta, cx<R> tb) {
    const cx<R> s0 = cfma(tb, g[db], g[0]);
    const cx<R> s1 = cfma(tb, g[da + db], g[da]);
    return cfma(ta, s1, s0);
  };
  cx<R> r[6];
  r[0] = caxpy(m0, f[0], vtx2face(hh, dyp, dzp, T[1], T[2]));
  r[1] = caxpy(m1, f[Nq], vtx2face(hh + Nq, dxp, dzp, T[0], T[2]));
  r[2] = caxpy(m2, f[2 * Nq], vtx2face(hh + 2 * Nq, dxp, dyp, T[0], T[1]));
  const cx<R>* hv = hh + 3 * Nq;
  r[3] = caxpy(n0, f[3 * Nq], cfma(T[0], hv[dxp], hv[0]));
  r[4] = caxpy(n1, f[4 * Nq], cfma(T[1], hv[Nq + dyp], hv[Nq]));
  r[5] = caxpy(n2, f[5 * Nq], cfma(T[2], hv[2 * Nq + dzp], hv[2 * Nq]));
  cx<R>* o = out + vec * stride + idx;
#pragma unroll
  for (int c = 0; c < 6; ++c) o[c * Nq] = r[c];
}

// ---------------------------------------------------------------------------
// Single-pass form: k_sweep reads the six spatial fields once and writes u',
// v' to a separate buffer, with no vertex scratch in global memory.  One CTA
// owns TY rows (all x) of a chunk of tz consecutive z-planes of one vector and
// sweeps through the chunk plane by plane, thread (r, x) on vertex row y0 + r
// (r = TY is the +y neighbour the scatter needs, evaluated but not written):
//   * the fields of a plane (rows y0-1 .. y0+TY) are staged in shared memory
//     by cp.async, the next plane in flight while this one is computed, the one
//     after it issued as soon as stage 1 has read its buffer;
//   * stage 1 gathers U, V and evaluates the vertex product.  Whatever the
//     next plane needs of this one is kept in registers, already summed over
//     its in-plane neighbours: s0 = u_0 + T_y^H u_0, s1 = u_1 + T_x^H u_1, u_5;
//   * the products that in-plane neighbours read go to shared memory (Hu, Hv_0,
//     Hv_1 and the real diagonals D; Hv_2 and a thread's own values stay in
//     registers);
//   * stage 2 finishes u'_2, v'_0, v'_1 of the plane, and u'_0, u'_1, v'_2 of
//     the plane below, from the partial sums carried in registers.
// Bound by the shared-memory pipe and by latency at two CTAs per SM.  Its
// first form kept two planes of H, D and three of fields in shared memory and
// re-read them (97 shared-memory accesses per vertex against 38 here, the
// pipe 66 % busy): fncB of 10 vectors at n = 60 257 -> 231 us, 8 at n = 48
// 126 -> 97, 3 at n = 50 70 -> 62 (complex64).  Three CTAs per SM (68
// registers) spill: 255 us at n = 60.
// ---------------------------------------------------------------------------
template <class R, int N> struct SweepShape {
  static constexpr int TY = N % 4 == 0 ? 4 : N % 5 == 0 ? 5 : N % 6 == 0 ? 6 : N % 3 == 0 ? 3 : N % 2 == 0 ? 2 : 1;
  static constexpr int FR = TY + 2;                       // staged field rows
  static constexpr int HR = TY + 1;                       // vertex rows
  static constexpr int TPB = ((HR * N + 31) / 32) * 32;
  // CTAs per SM: the 16384 registers of an SM's quarter hold 5 warps of 96
  // registers (complex64; complex128: 3 of 168).  Left to itself the compiler took
  // 130 for the general tensors at n = 30, 36, 50, 60, 64, one CTA fewer per SM
  // (fncB of ten vectors at n = 60 then 217 us, now 197; 16 at n = 30 50, now 44).
  static constexpr int WARPS = sizeof(R) == 4 ? 20 : 12;
  static constexpr int CTAS = WARPS >= TPB / 32 ? WARPS / (TPB / 32) : 1;
  static constexpr int F_ELEMS = 6 * FR * N;              // one staged plane (complex)
  static constexpr int H_ELEMS = 5 * HR * N;              // shared vertex values of one plane (complex)
  static constexpr int D_ELEMS = 5 * HR * N;              // shared diagonals of one plane (real)
  static constexpr int TAB_MAX = 8;                       // phases whose tensors are staged in shared memory
  static constexpr size_t SMEM = sizeof(cx<R>) * (2 * F_ELEMS + H_ELEMS) + sizeof(R) * (D_ELEMS + TAB_MAX * kStnGeneral);
  static constexpr int CPR = int(N * sizeof(cx<R>) / 16);  // 16-byte chunks per row
  // rows staged per plane: u_0, u_2, v_1 with the row below, the others without
  static constexpr int ROWS = 6 * FR - 3;
  static constexpr int CH = ROWS * CPR;                    // 16-byte chunks per staged plane
  static constexpr int NCH = (CH + TPB - 1) / TPB;         // chunks per thread
  static_assert((N * sizeof(cx<R>)) % 16 == 0, "rows must be whole 16-byte chunks");
  static_assert(TPB <= 1024 && N % TY == 0, "one thread per vertex of a plane's rows");
};

__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int K> __device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(K) : "memory");
}

template <class R, int N, int KIND>
__global__ void __launch_bounds__(SweepShape<R, N>::TPB, sizeof(R) == 4 && KIND == kMatGeneral ? SweepShape<R, N>::CTAS : 0)
k_sweep(const cx<R>* __restrict__ uv, cx<R>* __restrict__ out, PlanData<R> d, const uint8_t* __restrict__ phase,
        int nphase, const __grid_constant__ VecCtx ctx, long long stride, int tz, double2* __restrict__ wdot) {
  using SH = SweepShape<R, N>;
  constexpr int TY = SH::TY, FR = SH::FR, HR = SH::HR, TPB = SH::TPB, CPR = SH::CPR;
  constexpr int NN = N * N, Nq = NN * N;
  constexpr int EPC = 16 / int(sizeof(cx<R>));             // complex per 16-byte chunk
  constexpr int TS = stn_size(KIND);
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cx<R>* Fb = reinterpret_cast<cx<R>*>(smem_raw);            // [2][6][FR][N]
  cx<R>* H = Fb + 2 * SH::F_ELEMS;                           // [5][HR][N]  Hu_0..2, Hv_0, Hv_1
  R* Tb = reinterpret_cast<R*>(H + SH::H_ELEMS);             // [TAB_MAX][TS] vertex tensors
  R* D = Tb + SH::TAB_MAX * kStnGeneral;                     // [5][HR][N]  D0..4
  const int y0 = blockIdx.x * TY;
  const int z0 = blockIdx.y * tz;
  const int nz = min(tz, N - z0);                            // planes of this chunk
  const int vec = blockIdx.z;
  pdl_wait();
  if (ctx.active && !ctx.active[vec]) return;
  const int inst = vec_inst(ctx, vec);
  const int tid = threadIdx.x;
  const cx<R>* src = uv + vec * stride;
  cx<R>* dst = out + vec * stride;
  const cx<R> Tx = d.tau[inst * 3], Ty = d.tau[inst * 3 + 1], Tz = d.tau[inst * 3 + 2];
  // This thread's 16-byte chunks of a staged plane: shared-memory offset and
  // global offset within the plane, the same for every plane of the sweep.
  int soff[SH::NCH], goff[SH::NCH];
#pragma unroll
  for (int i = 0; i < SH::NCH; ++i) {
    const int c = tid + i * TPB;
    const int row = c / CPR, cc = c - row * CPR;
    const int q = row / (2 * FR - 1), rem = row - q * (2 * FR - 1);
    const int f = 2 * q + (rem >= FR ? 1 : 0);  // fields in the order 0 1 | 2 3 | 4 5
    const int r = rem < FR ? rem : rem - FR + 1;
    const int y = (y0 - 1 + r + N) % N;
    soff[i] = (f * FR + r) * N + cc * EPC;
    goff[i] = f * Nq + y * N + cc * EPC;
  }
  auto stage = [&](int s) {  // plane z0-1+s -> Fb[s % 2]
    const int z = (z0 - 1 + s + N) % N;
    cx<R>* F = Fb + (s & 1) * SH::F_ELEMS;
    const cx<R>* sp = src + z * NN;
#pragma unroll
    for (int i = 0; i < SH::NCH; ++i)
      if (tid + i * TPB < SH::CH) cp_async16(F + soff[i], sp + goff[i]);
    cp_async_commit();
  };
  stage(0);
  stage(1);
  const R* tab = nullptr;
  if constexpr (KIND != kMatField) {
    tab = d.stn + (size_t)inst * nphase * TS;
    if (nphase <= SH::TAB_MAX) {
      for (int i = tid; i < nphase * TS; i += TPB) Tb[i] = tab[i];
      tab = Tb;
    }
  }

  const int r = tid / N, x = tid - r * N;
  const bool act = tid < HR * N;   // stage 1
  const bool outp = tid < TY * N;  // stage 2
  const int xm = x == 0 ? N - 1 : x - 1, xp = x == N - 1 ? 0 : x + 1;
  const int row = (y0 + r) % N;
  const cx<R> TxTy = cmul(Tx, Ty);
  double acc = 0.0;  // sum of Re(conj(w) . out) over this CTA's outputs (wdot)
  int ph_next = 0;   // phase id of this thread's vertex on the next plane, loaded one step ahead
  if (KIND != kMatField && act) ph_next = __ldg(phase + z0 * NN + row * N + x);
  // carried from the plane below: in-plane sums s0, s1 of u_0, u_1, and the
  // partial outputs q0, q1, q5 with the fields f0, f1, f5 they still need
  cx<R> s0 = zero<R>(), s1 = zero<R>(), f0 = zero<R>(), f1 = zero<R>(), f5 = zero<R>();
  cx<R> q0 = zero<R>(), q1 = zero<R>(), q5 = zero<R>();
  for (int s = 0; s <= nz + 1; ++s) {
    if (s <= nz) cp_async_wait<1>();
    else cp_async_wait<0>();
    __syncthreads();  // plane s visible; H, D free again
    const cx<R>* F = Fb + (s & 1) * SH::F_ELEMS;
    auto at = [&](int f, int rr, int xx) { return F[(f * FR + rr) * N + xx]; };
    const int zc = (z0 - 1 + s + N) % N;
    cx<R> c[6], hu[3], hv[3];
    R dg[6];
    if (act) {
      // U_j = (I + T_a^H)(I + T_b^H) u_j, V_j = (I + T_j^H) v_j ; (T^H g)(r) = conj(T) g(r - e)
      c[0] = at(0, r + 1, x);
      c[1] = at(1, r + 1, x);
      c[5] = at(5, r + 1, x);
      const cx<R> p0 = cfmac(Ty, at(0, r, x), c[0]);
      const cx<R> p1 = cfmac(Tx, at(1, r + 1, xm), c[1]);
      if (s >= 1) {
        c[2] = at(2, r + 1, x);
        c[3] = at(3, r + 1, x);
        c[4] = at(4, r + 1, x);
        cx<R> U[3], V[3];
        U[0] = cfmac(Tz, s0, p0);
        U[1] = cfmac(Tz, s1, p1);
        U[2] = cfmac(TxTy, at(2, r, xm), cfmac(Ty, at(2, r, x), cfmac(Tx, at(2, r + 1, xm), c[2])));
        V[0] = cfmac(Tx, at(3, r + 1, xm), c[3]);
        V[1] = cfmac(Ty, at(4, r, x), c[4]);
        V[2] = cfmac(Tz, f5, c[5]);
        const int ph = ph_next;
        if (KIND != kMatField) ph_next = __ldg(phase + ((zc + 1) % N) * NN + row * N + x);
        vertex_product<R, KIND>(tab + ph * TS, d.fld + (zc * NN + row * N + x), Nq, d.gram, U, V, hu, hv, dg);
#pragma unroll
        for (int f = 0; f < 5; ++f) {
          H[(f * HR + r) * N + x] = f < 3 ? hu[f] : hv[f - 3];
          D[(f * HR + r) * N + x] = dg[f];
        }
      }
      s0 = p0;
      s1 = p1;
    }
    __syncthreads();  // H, D visible; the buffer of plane s free again
    if (s < nz) stage(s + 2);
    if (s >= 1 && outp) {
      auto h = [&](int f, int rr, int xx) { return H[(f * HR + rr) * N + xx]; };
      auto dd = [&](int f, int rr, int xx) { return D[(f * HR + rr) * N + xx]; };
      // u'_i = m_i u_i + (I+T_a)(I+T_b) Hu_i ; v'_i = n_i v_i + (I+T_i) Hv_i ; (T g)(r) = T g(r + e)
      const cx<R> g0 = cfma(Ty, h(0, r + 1, x), hu[0]);
      const cx<R> g1 = cfma(Tx, h(1, r, xp), hu[1]);
      const R e0 = dg[0] + dd(0, r + 1, x), e1 = dg[1] + dd(1, r, xp);
      cx<R>* op = dst + (y0 + r) * N + x;
      R a = 0;
      auto dotw = [&](cx<R> w, cx<R> o) { a = rfma(w.x, o.x, rfma(w.y, o.y, a)); };
      if (s >= 2) {  // the plane below: u'_0, u'_1, v'_2
        const int zo = (zc + N - 1) % N;
        const cx<R> o0 = caxpy(e0, f0, cfma(Tz, g0, q0));
        const cx<R> o1 = caxpy(e1, f1, cfma(Tz, g1, q1));
        const cx<R> o5 = caxpy(dg[5], f5, cfma(Tz, hv[2], q5));
        op[zo * NN] = o0;
        op[Nq + zo * NN] = o1;
        op[5 * Nq + zo * NN] = o5;
        if (wdot) {
          dotw(f0, o0);
          dotw(f1, o1);
          dotw(f5, o5);
        }
      }
      if (s <= nz) {
        const R m2 = (dg[2] + dd(2, r, xp)) + (dd(2, r + 1, x) + dd(2, r + 1, xp));
        const R n0 = dg[3] + dd(3, r, xp), n1 = dg[4] + dd(4, r + 1, x);
        const cx<R> o2 = caxpy(m2, c[2], cfma(TxTy, h(2, r + 1, xp), cfma(Ty, h(2, r + 1, x), cfma(Tx, h(2, r, xp), hu[2]))));
        const cx<R> o3 = caxpy(n0, c[3], cfma(Tx, h(3, r, xp), hv[0]));
        const cx<R> o4 = caxpy(n1, c[4], cfma(Ty, h(4, r + 1, x), hv[1]));
        op[2 * Nq + zc * NN] = o2;
        op[3 * Nq + zc * NN] = o3;
        op[4 * Nq + zc * NN] = o4;
        if (wdot) {
          dotw(c[2], o2);
          dotw(c[3], o3);
          dotw(c[4], o4);
        }
      }
      if (wdot) acc += double(a);
      q0 = caxpy(e0, c[0], g0);
      q1 = caxpy(e1, c[1], g1);
      q5 = caxpy(dg[5], c[5], hv[2]);
      f0 = c[0];
      f1 = c[1];
    }
    if (act) f5 = c[5];
  }
  if (wdot) {
    // one partial per CTA: [vec][blockIdx.y][blockIdx.x]
    __shared__ double red[32];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
    if ((tid & 31) == 0) red[tid >> 5] = acc;
    __syncthreads();
    if (tid < 32) {
      double v = tid < (TPB + 31) / 32 ? red[tid] : 0.0;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
      if (tid == 0)
        wdot[(long long)vec * gridDim.x * gridDim.y + blockIdx.y * gridDim.x + blockIdx.x] = make_double2(v, 0.0);
    }
  }
}

// f(integral_constant<KIND>) for the plan's kind of vertex tensors.
template <class R, class F> inline cudaError_t with_kind(const PlanData<R>& d, F&& f) {
  switch (d.kind) {
    case kMatField: return f(std::integral_constant<int, kMatField>{});
    case kMatChiral: return f(std::integral_constant<int, kMatChiral>{});
    default: return f(std::integral_constant<int, kMatGeneral>{});
  }
}

// z-planes per CTA of k_sweep for sub-batches of nv vectors: the chunk count
// with the least (waves of resident CTAs) x (planes a CTA steps through; its
// halo planes cost about 1.5).  One vector of a small grid takes one or two
// planes per CTA (n = 24: 12 planes in series took 19 us of a 35 us fncB),
// full batches long chunks.  The count of resident CTAs has to be the real one:
// 4 vectors at n = 40 in 400 CTAs, where 304 are resident, took 15.6 us, 11.3 in 280.
template <class R, int N> inline int sweep_planes(const Plan& P, int nv) {
  using SH = SweepShape<R, N>;
  const int per_sm = std::max<int>(1, std::min<int>(SH::CTAS, int((227u << 10) / (SH::SMEM + 1024))));
  const long long slots = (long long)per_sm * P.sms;
  int best = N;
  double cost = 1e300;
  for (int c = 1; c <= N; ++c) {
    const int tz = (N + c - 1) / c;
    const long long ctas = (long long)(N / SH::TY) * ((N + tz - 1) / tz) * std::max(1, nv);
    const double k = double((ctas + slots - 1) / slots) * (tz + 1.5);
    if (k < cost - 1e-9) {
      cost = k;
      best = tz;
    }
  }
  return best;
}

// Out of place: out = [M J^H; J N] w on 6-field vectors (stride 6*Nq).
// wdot (may be null): per-CTA partial sums of Re(w^H out), sweep_partials_n
// of them per vector; tz: sweep_planes of the batch.
template <class R, int N>
cudaError_t sweep_n(const Plan& P, const cx<R>* w, cx<R>* out, int nvec, const VecCtx& ctx, cudaStream_t st, int tz,
                    double2* wdot = nullptr) {
  using SH = SweepShape<R, N>;
  const PlanData<R>& d = pdata<R>(P);
  return with_kind<R>(d, [&](auto kc) -> cudaError_t {
    return launch<k_sweep<R, N, decltype(kc)::value>>(dim3(N / SH::TY, (N + tz - 1) / tz, nvec), SH::TPB, SH::SMEM,
                                                          st, w, out, d, P.d_phase, P.nphase, ctx, 6LL * N * N * N, tz,
                                                          wdot);
  });
}

template <class R, int N> int sweep_partials_n(int tz) { return (N / SweepShape<R, N>::TY) * ((N + tz - 1) / tz); }

// The two-kernel form: out = [M J^H; J N] w on 6-field vectors (stride 6*Nq;
// out may be w), scratch h of the same size, tpb threads per block (128, 256
// or 512).  bloch: fields in the Bloch frame (phases at the wraps only)
// instead of the periodic one.
template <class R, int N>
cudaError_t stencil_n(const Plan& P, const cx<R>* w, cx<R>* out, cx<R>* h, int nvec, const VecCtx& ctx,
                      cudaStream_t st, int tpb, bool bloch) {
  constexpr int Nq = N * N * N;
  if (tpb != 64 && tpb != 128 && tpb != 512) tpb = 256;
  const dim3 g((Nq + tpb - 1) / tpb, nvec);
  const PlanData<R>& d = pdata<R>(P);
  return with_kind<R>(d, [&](auto kc) -> cudaError_t {
    constexpr int K = decltype(kc)::value;
    cudaError_t e = launch<k_vertex<R, N, K>>(g, tpb, 0, st, w, h, d, P.d_phase, P.nphase, ctx, 6LL * Nq, bloch);
    if (e != cudaSuccess) return e;
    return launch<k_faceedge<R, N, K>>(g, tpb, 0, st, w, h, out, d, P.d_phase, P.nphase, ctx, 6LL * Nq, bloch);
  });
}

}  // namespace detail
}  // namespace fame

// Preconditioner of the conjugate-gradient solves with B (fncinvB).
//
// For a homogeneous medium every Bloch shift is diagonal in the frequency
// basis (T_d <-> t_d = exp(i(2 pi k_d + theta_d)/n) = 1 + lambda_d/n), so
// fncB reduces to one 4x4 Hermitian block per frequency voxel:
//   B0(k) = Pi(k)^H G(k) Pi(k),   Pi = blkdiag([-conj(Pi2) conj(Pi1)], [Pi1 Pi2])
// with G(k) the 6x6 material symbol of the interpolated operators
// (IntCovarForm*_vertex*.m): lumped diagonals Re Mh_ii, Re Nh_ii, and
//   M_ij: c_a c_b Mh_ij conj(c_a' c_b')/16 , N_ij: c_i Nh_ij conj(c_j)/4 ,
//   J_ij: c_i J_ij conj(c_a' c_b')/8        (c_d = 1 + t_d).
// Using the volume-averaged vertex tensors of the actual crystal, M = B0^{-1}
// is a cheap spectrally close approximation of B^{-1}; the CG iteration count
// drops by more than half on the woodpile.  The solution of B y = x does not
// depend on it.
#include "fncb_impl.cuh"
#include "krylov.h"
#include "launch.h"

namespace fame {
namespace {

__device__ __forceinline__ double2 dmk(double a, double b) { return make_double2(a, b); }

// Complex slots per voxel of the stored inverse blocks (the four real
// diagonal entries packed in two).
constexpr int kPcSlots = 8;

// FP64-rate-bound, once per plan: some 670 operations per voxel, with the
// Hermitian halves computed once and L D L^H in place of a Gauss-Jordan of the
// full block and its identity (8 instances at n = 48 2.3 -> 1.0 ms).
__global__ void __launch_bounds__(128)
k_precond_build64(const double2* __restrict__ lam_all, const double2* __restrict__ avg_all, int n, double2* pc64,
                  float2* pc32) {
  const long long Nq = (long long)n * n * n;
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int inst = blockIdx.y;
  if (idx >= Nq) return;
  const int i1 = int(idx % n), i2 = int((idx / n) % n), i3 = int(idx / ((long long)n * n));
  const double2* lam = lam_all + (long long)inst * 3 * n;
  const double2 L[3] = {lam[i1], lam[n + i2], lam[2 * n + i3]};
  // cv_i = c_i / 2, cu_i = c_a c_b / 4 of the two other axes
  double2 cv[3], cu[3];
  const double rn = 0.5 / n;
#pragma unroll
  for (int d = 0; d < 3; ++d) cv[d] = dmk(rfma(L[d].x, rn, 1.0), L[d].y * rn);
#pragma unroll
  for (int d = 0; d < 3; ++d) cu[d] = cmul(cv[d == 0 ? 1 : 0], cv[d == 2 ? 1 : 2]);
  const double2* T = avg_all + (long long)inst * 27;
  const double2* Nh = T;
  const double2* Mh = T + 9;
  const double2* J = T + 18;
  // columns of Pi: u-side e0 = -conj(Pi2), e1 = conj(Pi1); v-side f0 = Pi1, f1 = Pi2
  const detail::PiBlock<double> P = detail::pi_block<double>(L[0], L[1], L[2]);
  double2 e[2][3];
#pragma unroll
  for (int r = 0; r < 3; ++r) {
    e[0][r] = cneg(cconj(P.p2[r]));
    e[1][r] = cconj(P.p1[r]);
  }
  const double2* f[2] = {P.p1, P.p2};
  // G[r][q] of a Hermitian symbol with scales s: s_r t_rq conj(s_q), real diagonal t_rr
  auto symbol = [](const double2* t, const double2* s, double2 (&G)[3][3]) {
#pragma unroll
    for (int r = 0; r < 3; ++r) {
      G[r][r] = dmk(t[4 * r].x, 0.0);
#pragma unroll
      for (int q = r + 1; q < 3; ++q) {
        G[r][q] = cmulc(s[q], cmul(s[r], t[3 * r + q]));
        G[q][r] = cconj(G[r][q]);
      }
    }
  };
  auto row = [](const double2 (&g)[3], const double2* v, int real) {  // sum_q g_q v_q; g[real] is real
    double2 w = dmk(0.0, 0.0);
#pragma unroll
    for (int q = 0; q < 3; ++q) w = q == real ? caxpy(g[q].x, v[q], w) : cfma(g[q], v[q], w);
    return w;
  };
  auto dot = [](const double2* a, const double2 (&g)[3]) {
    return cfmac(a[2], g[2], cfmac(a[1], g[1], cmulc(a[0], g[0])));
  };
  auto dotr = [](const double2* a, const double2 (&g)[3]) {
    double w = 0.0;
#pragma unroll
    for (int r = 0; r < 3; ++r) w = rfma(a[r].x, g[r].x, rfma(a[r].y, g[r].y, w));
    return w;
  };
  // lower triangle of B0 in the order e0, e1, f0, f1
  double b00, b11, b22, b33;
  double2 b10, b32, bvu[2][2];
  double2 g0[3], g1[3], G[3][3];
  symbol(Mh, cu, G);
#pragma unroll
  for (int r = 0; r < 3; ++r) {
    g0[r] = row(G[r], e[0], r);
    g1[r] = row(G[r], e[1], r);
  }
  b00 = dotr(e[0], g0);
  b10 = dot(e[1], g0);
  b11 = dotr(e[1], g1);
  symbol(Nh, cv, G);
#pragma unroll
  for (int r = 0; r < 3; ++r) {
    g0[r] = row(G[r], f[0], r);
    g1[r] = row(G[r], f[1], r);
  }
  b22 = dotr(f[0], g0);
  b32 = dot(f[1], g0);
  b33 = dotr(f[1], g1);
#pragma unroll
  for (int r = 0; r < 3; ++r) {
#pragma unroll
    for (int q = 0; q < 3; ++q) G[r][q] = cmulc(cu[q], cmul(cv[r], J[3 * r + q]));
    g0[r] = row(G[r], e[0], -1);
    g1[r] = row(G[r], e[1], -1);
  }
#pragma unroll
  for (int a = 0; a < 2; ++a) {
    bvu[a][0] = dot(f[a], g0);
    bvu[a][1] = dot(f[a], g1);
  }
  double2 b20 = bvu[0][0], b21 = bvu[0][1], b30 = bvu[1][0], b31 = bvu[1][1];
  // B0 = L D L^H: a -= l conj(b) with l = b'/d
  auto sub = [](double2 l, double2 b, double2 a) { return cfmac(b, cneg(l), a); };
  auto subr = [](double2 l, double2 b, double a) { return rfma(-l.x, b.x, rfma(-l.y, b.y, a)); };
  const double r0 = 1.0 / b00;
  const double2 l10 = cscale(b10, r0), l20 = cscale(b20, r0), l30 = cscale(b30, r0);
  b11 = subr(l10, b10, b11);
  b21 = sub(l20, b10, b21);
  b31 = sub(l30, b10, b31);
  b22 = subr(l20, b20, b22);
  b32 = sub(l30, b20, b32);
  b33 = subr(l30, b30, b33);
  const double r1 = 1.0 / b11;
  const double2 l21 = cscale(b21, r1), l31 = cscale(b31, r1);
  b22 = subr(l21, b21, b22);
  b32 = sub(l31, b21, b32);
  b33 = subr(l31, b31, b33);
  const double r2 = 1.0 / b22;
  const double2 l32 = cscale(b32, r2);
  b33 = subr(l32, b32, b33);
  const double r3 = 1.0 / b33;
  // X = L^{-1}, M = X^H D^{-1} X
  const double2 x10 = cneg(l10), x21 = cneg(l21), x32 = cneg(l32);
  const double2 x20 = cneg(cfma(l21, x10, l20));
  const double2 x31 = cneg(cfma(l32, x21, l31));
  const double2 x30 = cneg(cfma(l32, x20, cfma(l31, x10, l30)));
  const double2 w30 = cscale(x30, r3), w31 = cscale(x31, r3), w32 = cscale(x32, r3);
  const double2 w20 = cscale(x20, r2), w21 = cscale(x21, r2), w10 = cscale(x10, r1);
  auto add = [](double2 w, double2 x, double a) { return rfma(w.x, x.x, rfma(w.y, x.y, a)); };
  double m00 = add(w30, x30, add(w20, x20, add(w10, x10, r0)));
  double m11 = add(w31, x31, add(w21, x21, r1));
  double m22 = add(w32, x32, r2);
  double m33 = r3;
  double2 m01 = cfmac(w30, x31, cfmac(w20, x21, cconj(w10)));
  double2 m02 = cfmac(w30, x32, cconj(w20));
  double2 m03 = cconj(w30);
  double2 m12 = cfmac(w31, x32, cconj(w21));
  double2 m13 = cconj(w31), m23 = cconj(w32);
  if (!(b00 > 0.0 && b11 > 0.0 && b22 > 0.0 && b33 > 0.0)) {  // not positive definite (non-physical material): identity
    m00 = m11 = m22 = m33 = 1.0;
    m01 = m02 = m03 = m12 = m13 = m23 = dmk(0.0, 0.0);
  }
  // packed: (m00, m11) | (m22, m33) | m01 | m02 | m03 | m12 | m13 | m23
  const double2 v[kPcSlots] = {dmk(m00, m11), dmk(m22, m33), m01, m02, m03, m12, m13, m23};
#pragma unroll
  for (int k = 0; k < kPcSlots; ++k) {
    const long long o = ((long long)inst * kPcSlots + k) * Nq + idx;
    if (pc64) pc64[o] = v[k];
    if (pc32) pc32[o] = make_float2(float(v[k].x), float(v[k].y));
  }
}

// The inverse block of one voxel.
template <class R> struct Block4 {
  cx<R> s[kPcSlots];
};
template <class R>
__device__ __forceinline__ Block4<R> load_block(const cx<R>* __restrict__ pc, long long Nq, long long idx) {
  Block4<R> b;
#pragma unroll
  for (int e = 0; e < kPcSlots; ++e) b.s[e] = pc[e * Nq + idx];
  return b;
}
// z = M r for the 4 components of one voxel
template <class R>
__device__ __forceinline__ void mvec4(const Block4<R>& b, const cx<R> r[4], cx<R> z[4]) {
  const R m00 = b.s[0].x, m11 = b.s[0].y, m22 = b.s[1].x, m33 = b.s[1].y;
  const cx<R> m01 = b.s[2], m02 = b.s[3], m03 = b.s[4], m12 = b.s[5], m13 = b.s[6], m23 = b.s[7];
  z[0] = cfma(m03, r[3], cfma(m02, r[2], cfma(m01, r[1], cscale(r[0], m00))));
  z[1] = cfma(m13, r[3], cfma(m12, r[2], cfmac(m01, r[0], cscale(r[1], m11))));
  z[2] = cfma(m23, r[3], cfmac(m12, r[1], cfmac(m02, r[0], cscale(r[2], m22))));
  z[3] = cfmac(m23, r[2], cfmac(m13, r[1], cfmac(m03, r[0], cscale(r[3], m33))));
}

constexpr int kThreads = 256;

// Block-wide sum, valid in thread 0 (block_sum2 of krylov_kernels.cu).
__device__ __forceinline__ double2 block_sum2b(double2 v) {
  __shared__ double2 sh[kThreads];
  sh[threadIdx.x] = v;
  __syncthreads();
  if (threadIdx.x < 32) {
#pragma unroll
    for (int k = 1; k < kThreads / 32; ++k) {
      v.x += sh[threadIdx.x + 32 * k].x;
      v.y += sh[threadIdx.x + 32 * k].y;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      v.x += __shfl_down_sync(0xffffffffu, v.x, o);
      v.y += __shfl_down_sync(0xffffffffu, v.y, o);
    }
  }
  return v;
}

// The start of a CG solve in one pass (pcg_start): reads b and the block,
// writes x, r, p (and z).
template <class R>
__global__ void __launch_bounds__(kThreads)
k_pcg_start(const cx<R>* __restrict__ b, cx<R>* __restrict__ x, cx<R>* __restrict__ r, cx<R>* __restrict__ z,
            cx<R>* __restrict__ p, const cx<R>* __restrict__ pc_all, const __grid_constant__ VecCtx ctx, long long Nq,
            double2* __restrict__ partial) {
  const int vec = blockIdx.y;
  const int nblk = gridDim.x;
  double2* out = partial + (long long)vec * nblk + blockIdx.x;
  pdl_wait();
  if (ctx.active && !ctx.active[vec]) {
    if (threadIdx.x == 0) *out = make_double2(0.0, 0.0);
    return;
  }
  const cx<R>* pc = pc_all ? pc_all + (long long)vec_inst(ctx, vec) * kPcSlots * Nq : nullptr;
  const long long o = vec * 4 * Nq;
  RunSum<R> srz, srr;
  const long long chunk = (Nq + nblk - 1) / nblk, end = min(Nq, (blockIdx.x + 1) * chunk);
  for (long long i = blockIdx.x * chunk + threadIdx.x; i < end; i += kThreads) {
    cx<R> rv[4], zv[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) zv[c] = rv[c] = b[o + c * Nq + i];
    if (pc) mvec4<R>(load_block<R>(pc, Nq, i), rv, zv);
    R trz = 0, trr = 0;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const long long k = o + c * Nq + i;
      x[k] = zero<R>();
      r[k] = rv[c];
      p[k] = zv[c];
      if (pc) z[k] = zv[c];
      trz = rfma(rv[c].x, zv[c].x, rfma(rv[c].y, zv[c].y, trz));
      trr = rfma(rv[c].x, rv[c].x, rfma(rv[c].y, rv[c].y, trr));
    }
    srz.add(trz);
    srr.add(trr);
  }
  double2 s = block_sum2b(make_double2(srz.value(), srr.value()));
  if (threadIdx.x == 0) *out = s;
}

// CG update of one vector's chunk of voxels per CTA: r -= a q, z = M r and the
// partial sums (x += a p is left to k_cg_dir, which reads p anyway).  HBM-bound
// on large batches, latency-bound on small ones, so that
//   * a CTA takes one contiguous chunk, and the CTAs of a launch are whole
//     multiples of what fits the SMs (dot_blocks);
//   * the loads of the first elements are issued before the step length, which
//     every CTA reduces from the stencil pass's partials, is waited for;
//   * complex64 moves two voxels per 16-byte access.
// 4 vectors at n = 40 (complex64) 20 -> 11 us, 2 at n = 30 (complex128) 26 -> 12,
// 8 at n = 48 (complex64) 44 -> 30 (184 MB, 6.2 TB/s).
template <class R>
__global__ void __launch_bounds__(kThreads, sizeof(R) == 4 ? 2 : 1)
k_pcg_update(cx<R>* __restrict__ r, cx<R>* __restrict__ z, const cx<R>* __restrict__ q,
             const cx<R>* __restrict__ pc_all, const __grid_constant__ VecCtx ctx, long long Nq,
             double2* __restrict__ partial, CgAlpha ca) {
  constexpr int U = 16 / sizeof(cx<R>);  // voxels per 16-byte access (n^3 is even)
  struct alignas(16) Pack {
    cx<R> e[U];
  };
  const int vec = blockIdx.y;
  const int nblk = gridDim.x;
  double2* out = partial + (long long)vec * nblk + blockIdx.x;
  __shared__ int s_act;
  __shared__ double s_alpha;
  pdl_wait();
  // one read per CTA: CTA 0 may clear the flag while others start
  if (threadIdx.x == 0) s_act = ctx.active ? ctx.active[vec] : 1;
  __syncthreads();
  if (!s_act) {
    if (threadIdx.x == 0) {
      *out = make_double2(0.0, 0.0);
      if (blockIdx.x == 0) ca.go[vec] = 0;
    }
    return;
  }
  const cx<R>* pc = pc_all + (long long)vec_inst(ctx, vec) * kPcSlots * Nq;
  const long long o = vec * 4 * Nq;
  const int np = int(Nq / U), chunk = (np + nblk - 1) / nblk;  // packs, packs per CTA
  const int end = min(np, (int(blockIdx.x) + 1) * chunk);
  int i = blockIdx.x * chunk + threadIdx.x;
  Pack qk[4], rk[4], bk[kPcSlots];
  auto load = [&](int j) {
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const long long k = o + c * Nq + (long long)j * U;
      qk[c] = *reinterpret_cast<const Pack*>(q + k);
      rk[c] = *reinterpret_cast<const Pack*>(r + k);
    }
#pragma unroll
    for (int c = 0; c < kPcSlots; ++c) bk[c] = *reinterpret_cast<const Pack*>(pc + c * Nq + (long long)j * U);
  };
  if (i < end) load(i);
  if (threadIdx.x < 32) {
    double sx = 0.0, sy = 0.0;
    for (int j = threadIdx.x; j < ca.nblk; j += 32) {
      const double2 t = ca.pq[(long long)vec * ca.nblk + j];
      sx += t.x;
      sy += t.y;
    }
#pragma unroll
    for (int w = 16; w > 0; w >>= 1) {
      sx += __shfl_down_sync(0xffffffffu, sx, w);
      sy += __shfl_down_sync(0xffffffffu, sy, w);
    }
    if (threadIdx.x == 0) {
      const bool ok = sx > 0.0 && isfinite(sx);
      const double av = ok ? ca.rho[vec] / sx : 0.0;
      s_alpha = av;
      if (blockIdx.x == 0) {
        ca.alpha[vec] = av;
        ca.go[vec] = ok;
        ca.dot[vec] = make_double2(sx, sy);
        if (!ok) {  // breakdown: B must be HPD
          ca.active[vec] = 0;
          ca.iters[vec] = -(ca.iters[vec] + 1);
        }
      }
    }
  }
  __syncthreads();
  const R a = R(s_alpha);
  RunSum<R> srz, srr;
  while (i < end) {
    Pack zk[4];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      cx<R> rv[4], zv[4];
      Block4<R> bl;
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        rk[c].e[u] = caxpy(-a, qk[c].e[u], rk[c].e[u]);
        rv[c] = rk[c].e[u];
      }
#pragma unroll
      for (int c = 0; c < kPcSlots; ++c) bl.s[c] = bk[c].e[u];
      mvec4<R>(bl, rv, zv);
      R trz = 0, trr = 0;
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        zk[c].e[u] = zv[c];
        trz = rfma(rv[c].x, zv[c].x, rfma(rv[c].y, zv[c].y, trz));
        trr = rfma(rv[c].x, rv[c].x, rfma(rv[c].y, rv[c].y, trr));
      }
      srz.add(trz);
      srr.add(trr);
    }
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const long long k = o + c * Nq + (long long)i * U;
      *reinterpret_cast<Pack*>(r + k) = rk[c];
      *reinterpret_cast<Pack*>(z + k) = zk[c];
    }
    i += kThreads;
    if (i < end) load(i);
  }
  double2 s = block_sum2b(make_double2(srz.value(), srr.value()));
  if (threadIdx.x == 0) *out = s;
}

}  // namespace

template <class R> PlanData<R>& pd_mut(Plan& P);
template <> PlanData<double>& pd_mut<double>(Plan& P) { return P.d64; }
template <> PlanData<float>& pd_mut<float>(Plan& P) { return P.d32; }

template <class R> cudaError_t build_precond(Plan& P, cudaStream_t st) {
  PlanData<R>& d = pd_mut<R>(P);
  if (d.pc) return cudaSuccess;
  cudaError_t e;
  if (!P.d_mat_avg) {
    e = cudaMalloc(&P.d_mat_avg, sizeof(double2) * 27 * P.nk);
    if (e != cudaSuccess) return e;
    e = cudaMemcpy(P.d_mat_avg, P.mat_avg.data(), sizeof(double2) * 27 * P.nk, cudaMemcpyHostToDevice);
    if (e != cudaSuccess) return e;
  }
  e = cudaMalloc(&d.pc, sizeof(cx<R>) * kPcSlots * (size_t)P.Nq * P.nk);
  if (e != cudaSuccess) return e;
  FAME_LAUNCHED(1);
  k_precond_build64<<<dim3((unsigned)((P.Nq + 127) / 128), P.nk), 128, 0, st>>>(
      P.d64.lam, P.d_mat_avg, P.n, sizeof(R) == 8 ? (double2*)d.pc : nullptr,
      sizeof(R) == 4 ? (float2*)d.pc : nullptr);
  return cudaGetLastError();
}

template <class R>
cudaError_t pcg_start(const Plan& P, bool precond, const cx<R>* b, cx<R>* x, cx<R>* r, cx<R>* z, cx<R>* p, int nvec,
                      const VecCtx& ctx, double2* partial, int nblk, cudaStream_t st) {
  const cx<R>* pc = precond ? detail::pdata<R>(P).pc : nullptr;
  return launch<k_pcg_start<R>>(dim3(nblk, nvec), kThreads, 0, st, b, x, r, z, p, pc, ctx, P.Nq, partial);
}

template <class R>
cudaError_t pcg_update(const Plan& P, cx<R>* r, cx<R>* z, const cx<R>* q, int nvec, const VecCtx& ctx,
                       double2* partial, int nblk, cudaStream_t st, const CgAlpha& ca) {
  const PlanData<R>& d = detail::pdata<R>(P);
  return launch<k_pcg_update<R>>(dim3(nblk, nvec), kThreads, 0, st, r, z, q, d.pc, ctx, P.Nq, partial, ca);
}

template cudaError_t build_precond<float>(Plan&, cudaStream_t);
template cudaError_t build_precond<double>(Plan&, cudaStream_t);
template cudaError_t pcg_start<float>(const Plan&, bool, const cx<float>*, cx<float>*, cx<float>*, cx<float>*, cx<float>*, int,
                                         const VecCtx&, double2*, int, cudaStream_t);
template cudaError_t pcg_start<double>(const Plan&, bool, const cx<double>*, cx<double>*, cx<double>*, cx<double>*, cx<double>*, int,
                                         const VecCtx&, double2*, int, cudaStream_t);
template cudaError_t pcg_update<float>(const Plan&, cx<float>*, cx<float>*, const cx<float>*, int, const VecCtx&,
                                       double2*, int, cudaStream_t, const CgAlpha&);
template cudaError_t pcg_update<double>(const Plan&, cx<double>*, cx<double>*, const cx<double>*, int, const VecCtx&,
                                        double2*, int, cudaStream_t, const CgAlpha&);

}  // namespace fame

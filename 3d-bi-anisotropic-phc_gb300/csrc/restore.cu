// Eigenvector restoration, ORGSEP residual and field maxima on the GPU.
//
// Eigen_Restoration_Chiral_no_inv.m:3-25: for x = [x1; x2],
//   [e; h] = -i [N J; J^H M] [Qr x2; Pr x1].
// With u = Pr x1, v = Qr x2 this is e = -i v', h = -i u' where [u'; v'] is the
// material operator of fncB applied to [u; v] (fncB.m:4-5): the first half of
// fncB and the stencil give it, in the periodic frame (the Bloch frame is
// S .* that, S the diagonal phase of MtxVecMul_FFT).
//
// EvaluteError_Chiral_no_inv.m:19 (ORGSEP):
//   || [N J; J^H M] [C^H h; -C e] - i omega [e; h] ||
// with C the explicit curl of @DistOp/C.m (forward differences with Bloch
// wrap, mesh length 1/n).  In the periodic frame each difference is
// n (tau_d f(r + e_d) - f(r)); the material product is again the stencil, on
// [u; v] = [-C e; C^H h], giving [h-row; e-row] = [u''; v''].
//
// Fig6cd_plot_max_field.m:58-69: max over components of |e_c| and |h_c|,
// optionally only at vertices outside the inclusion (phase id 0).
#include <cmath>
#include <vector>

#include "fame_internal.h"
#include "launch.h"

namespace fame {
namespace {

constexpr int kT = 128;

// The fields [e; h] = [-i v'; -i u'] are read from the stencil output w = [u'; v']
// where they are needed (a swap of components; no pass of their own).
__device__ __forceinline__ double2 field_of(double2 wv) { return cmul_i<-1>(wv); }

// Y = [-C e; C^H h] / n (periodic frame): D_d f = n (tau_d f(r+e_d) - f(r)),
// D_d^H g = n (conj(tau_d) g(r-e_d) - g(r)); the mesh factor n is applied with the
// residual (the material product in between is linear).  FP64-rate-bound: 60
// operations per voxel (8 vectors at n = 40: 106 us with the differences scaled
// one by one, 58 now).
__global__ void __launch_bounds__(kT)
k_curl_pair(const double2* __restrict__ w, double2* __restrict__ y, PlanData<double> d,
            const __grid_constant__ VecCtx ctx, int n) {
  const long long Nq = (long long)n * n * n;
  const int idx = blockIdx.x * kT + threadIdx.x;
  const int vec = blockIdx.y;
  pdl_wait();
  if (idx >= Nq) return;
  const int inst = vec_inst(ctx, vec);
  const int i1 = idx % n, i2 = (idx / n) % n, i3 = idx / (n * n);
  const int sy = n, sz = n * n;
  const int dxp = i1 == n - 1 ? -(n - 1) : 1, dxm = i1 == 0 ? n - 1 : -1;
  const int dyp = i2 == n - 1 ? -(n - 1) * sy : sy, dym = i2 == 0 ? (n - 1) * sy : -sy;
  const int dzp = i3 == n - 1 ? -(n - 1) * sz : sz, dzm = i3 == 0 ? (n - 1) * sz : -sz;
  const double2* tau = d.tau + inst * 3;
  const double2 tx = tau[0], ty = tau[1], tz = tau[2];
  const double2* h = w + vec * 6 * Nq + idx;  // u': h_c = -i u'_c
  const double2* e = h + 3 * Nq;              // v': e_c = -i v'_c
  auto at = [&](const double2* f, int c, int o) { return field_of(f[c * Nq + o]); };
  // D_a f - D_b g = (ta f(+a) - f) - (tb g(+b) - g)
  auto two = [&](double2 fp, double2 f, double2 ta, double2 gp, double2 g, double2 tb) {
    return cfma(ta, fp, cfma(cneg(tb), gp, csub(g, f)));
  };
  auto two_h = [&](double2 fm, double2 f, double2 ta, double2 gm, double2 g, double2 tb) {
    return cfmac(ta, fm, cfmac(cneg(tb), gm, csub(g, f)));
  };
  const double2 e0 = at(e, 0, 0), e1 = at(e, 1, 0), e2 = at(e, 2, 0);
  const double2 h0 = at(h, 0, 0), h1 = at(h, 1, 0), h2 = at(h, 2, 0);
  double2* o = y + vec * 6 * Nq + idx;
  // -C e = [Dz e1 - Dy e2; Dx e2 - Dz e0; Dy e0 - Dx e1]
  o[0] = two(at(e, 1, dzp), e1, tz, at(e, 2, dyp), e2, ty);
  o[Nq] = two(at(e, 2, dxp), e2, tx, at(e, 0, dzp), e0, tz);
  o[2 * Nq] = two(at(e, 0, dyp), e0, ty, at(e, 1, dxp), e1, tx);
  // C^H h = [Dz^H h1 - Dy^H h2; Dx^H h2 - Dz^H h0; Dy^H h0 - Dx^H h1]
  o[3 * Nq] = two_h(at(h, 1, dzm), h1, tz, at(h, 2, dym), h2, ty);
  o[4 * Nq] = two_h(at(h, 2, dxm), h2, tx, at(h, 0, dzm), h0, tz);
  o[5 * Nq] = two_h(at(h, 0, dym), h0, ty, at(h, 1, dxm), h1, tx);
}

// Per block: sum |n v'' - i w e|^2 + |n u'' - i w h|^2, max |e_c|^2, max |h_c|^2
// (masked to phase id 0 when outside_only).  (The squares are compared and the
// root of their maximum taken once: with six FP64 roots per voxel 104 us for 8
// vectors at n = 40, 67 now.)
__global__ void __launch_bounds__(kT)
k_orgsep(const double2* __restrict__ y, const double2* __restrict__ w, const double* __restrict__ om,
         const uint8_t* __restrict__ phase, int outside_only, long long Nq, double mesh, double* __restrict__ part) {
  const int vec = blockIdx.y;
  pdl_wait();
  const double om_v = om[vec];
  double s = 0.0, me = 0.0, mh = 0.0;
  const long long chunk = (Nq + gridDim.x - 1) / gridDim.x, end = min(Nq, (blockIdx.x + 1) * chunk);
  for (long long idx = blockIdx.x * chunk + threadIdx.x; idx < end; idx += kT) {
    const double2* yv = y + vec * 6 * Nq + idx;
    const double2* wv = w + vec * 6 * Nq + idx;
    const bool use = !outside_only || phase[idx] == 0;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const double2 ec = field_of(wv[(3 + c) * Nq]), hc = field_of(wv[c * Nq]);
      const double2 r1 = caxpyi(-om_v, ec, cscale(yv[(3 + c) * Nq], mesh));
      const double2 r2 = caxpyi(-om_v, hc, cscale(yv[c * Nq], mesh));
      s = fma(r1.x, r1.x, fma(r1.y, r1.y, fma(r2.x, r2.x, fma(r2.y, r2.y, s))));
      if (use) {
        me = fmax(me, ec.x * ec.x + ec.y * ec.y);
        mh = fmax(mh, hc.x * hc.x + hc.y * hc.y);
      }
    }
  }
  __shared__ double rs[kT], re[kT], rh[kT];
  rs[threadIdx.x] = s;
  re[threadIdx.x] = me;
  rh[threadIdx.x] = mh;
  __syncthreads();
  if (threadIdx.x < 32) {
#pragma unroll
    for (int k = 1; k < kT / 32; ++k) {
      s += rs[threadIdx.x + 32 * k];
      me = fmax(me, re[threadIdx.x + 32 * k]);
      mh = fmax(mh, rh[threadIdx.x + 32 * k]);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      s += __shfl_down_sync(0xffffffffu, s, o);
      me = fmax(me, __shfl_down_sync(0xffffffffu, me, o));
      mh = fmax(mh, __shfl_down_sync(0xffffffffu, mh, o));
    }
    if (threadIdx.x == 0) {
      double* p = part + ((long long)vec * gridDim.x + blockIdx.x) * 3;
      p[0] = s;
      p[1] = me;
      p[2] = mh;
    }
  }
}

// E = S .* e, H = S .* h (Bloch frame, the reference's layout: 3Nq each).
__global__ void __launch_bounds__(kT)
k_to_bloch(const double2* __restrict__ w, double2* __restrict__ E, double2* __restrict__ H, PlanData<double> d,
           const __grid_constant__ VecCtx ctx, int n) {
  const long long Nq = (long long)n * n * n;
  const int idx = blockIdx.x * kT + threadIdx.x;
  const int vec = blockIdx.y;
  pdl_wait();
  if (idx >= Nq) return;
  const int i1 = idx % n, i2 = (idx / n) % n, i3 = idx / (n * n);
  const double2* S = d.sxyz + (long long)vec_inst(ctx, vec) * 3 * n;
  const double2 s = cmul(cmul(S[i1], S[n + i2]), S[2 * n + i3]);
  const double2* src = w + vec * 6 * Nq + idx;
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    if (E) E[vec * 3 * Nq + c * Nq + idx] = cmul(s, field_of(src[(3 + c) * Nq]));
    if (H) H[vec * 3 * Nq + c * Nq + idx] = cmul(s, field_of(src[c * Nq]));
  }
}

}  // namespace
}  // namespace fame

using namespace fame;

extern "C" int fame_restore(fame_plan_t h, int nvec, const int* inst, const void* x, const double* omega, void* E,
                            void* H, double* res_orgsep, double* max_e, double* max_h, int outside_only) {
  if (!h) return FAME_ERR_BAD_ARG;
  Plan& P = h->P;
  if (nvec < 1 || !x || !omega) return fail(&P, FAME_ERR_BAD_ARG, "fame_restore: bad argument");
  if (inst)
    for (int v = 0; v < nvec; ++v)
      if (inst[v] < 0 || inst[v] >= P.nk) return fail(&P, FAME_ERR_BAD_ARG, "fame_restore: bad instance");
  cudaStream_t st = P.stream;
  const long long Nq = P.Nq;
  cudaError_t e = ensure_work(P, (size_t)nvec);
  if (e != cudaSuccess) return cuda_fail(&P, e, "fame_restore work");
  double2* w0 = (double2*)P.d_work;
  double2* w1 = w0 + (size_t)nvec * 6 * Nq;
  const size_t six = sizeof(double2) * 6 * (size_t)Nq * nvec;
  double2* y = (double2*)workspace(P, 45, six, &e);  // the curl pair and its material product
  if (e != cudaSuccess) return cuda_fail(&P, e, "fame_restore scratch");
  VecCtx ctx;
  ctx.nk = P.nk;
  if (inst && !small_inst(ctx, inst, nvec)) {
    int* d_inst = (int*)workspace(P, 46, sizeof(int) * nvec, &e);
    if (e == cudaSuccess) e = h2d_async(P, d_inst, inst, sizeof(int) * nvec);
    if (e != cudaSuccess) return cuda_fail(&P, e, "fame_restore inst");
    ctx.inst = d_inst;
  }
  const dim3 g((unsigned)((Nq + kT - 1) / kT), (unsigned)nvec);
#define RS_CK(expr, what)                              \
  do {                                                 \
    cudaError_t e_ = (expr);                           \
    if (e_ != cudaSuccess) return cuda_fail(&P, e_, what); \
  } while (0)
  RS_CK(launch_fields_inv<double>(P, (const double2*)x, w0, nvec, ctx, st), "fame_restore fields");
  RS_CK(launch_stencil<double>(P, w0, w0, w1, nvec, ctx, st), "fame_restore material");
  const bool want_res = res_orgsep || max_e || max_h;
  const int nblk = 152;
  double* part = nullptr;
  if (want_res) {
    double* d_om = (double*)workspace(P, 47, sizeof(double) * nvec, &e);
    if (e == cudaSuccess) e = h2d_async(P, d_om, omega, sizeof(double) * nvec);
    RS_CK(e, "fame_restore omega");
    RS_CK(launch<k_curl_pair>(g, kT, 0, st, w0, y, P.d64, ctx, P.n), "k_curl_pair");
    RS_CK(launch_stencil<double>(P, y, y, w1, nvec, ctx, st), "fame_restore residual material");
    part = (double*)workspace(P, 48, sizeof(double) * 3 * nblk * nvec, &e);
    RS_CK(e, "fame_restore partials");
    RS_CK(launch<k_orgsep>(dim3(nblk, nvec), kT, 0, st, y, w0, d_om, P.d_phase, outside_only, Nq, double(P.n), part),
          "k_orgsep");
  }
  if (E || H) RS_CK(launch<k_to_bloch>(g, kT, 0, st, w0, (double2*)E, (double2*)H, P.d64, ctx, P.n), "k_to_bloch");
  if (want_res) {
    std::vector<double> hp((size_t)3 * nblk * nvec);
    RS_CK(cudaMemcpyAsync(hp.data(), part, sizeof(double) * hp.size(), cudaMemcpyDeviceToHost, st), "orgsep d2h");
    RS_CK(cudaStreamSynchronize(st), "orgsep sync");
    for (int v = 0; v < nvec; ++v) {
      double s = 0.0, me = 0.0, mh = 0.0;
      for (int b = 0; b < nblk; ++b) {
        const double* p = &hp[((size_t)v * nblk + b) * 3];
        s += p[0];
        me = std::fmax(me, p[1]);
        mh = std::fmax(mh, p[2]);
      }
      if (res_orgsep) res_orgsep[v] = std::sqrt(s);
      if (max_e) max_e[v] = std::sqrt(me);
      if (max_h) max_h[v] = std::sqrt(mh);
    }
  }
#undef RS_CK
  return FAME_OK;
}

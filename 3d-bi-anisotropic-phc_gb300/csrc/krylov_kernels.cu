// Vector kernels of the Krylov glue: batched complex dot products with FP64
// accumulation, the fused conjugate-gradient updates of fncinvB (pcg), and
// the block Gram-Schmidt / restart products of the Lanczos band solver.
// Every kernel works on a batch of vectors, one vector per k-point instance,
// and skips vectors whose `active` flag is 0.
#include "krylov.h"
#include "launch.h"

namespace fame {
namespace {

constexpr int kRedThreads = 256;

// Block-wide sum of a (double re, double im) pair; result valid in thread 0.
// Through shared memory by one warp: 24 FP64 warp instructions instead of the
// 90 of a shuffle tree in every warp (each takes the SM's FP64 pipe for 16
// cycles, and small launches are mostly their reductions).
__device__ __forceinline__ double2 block_sum2(double2 v) {
  __shared__ double2 sh[kRedThreads];
  sh[threadIdx.x] = v;
  __syncthreads();
  if (threadIdx.x < 32) {
#pragma unroll
    for (int k = 1; k < kRedThreads / 32; ++k) {
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

// Sum of n partials, by the first warp of the block; valid in thread 0.
__device__ __forceinline__ double2 warp_sum2(const double2* __restrict__ q, int n) {
  double2 s = make_double2(0.0, 0.0);
  if (threadIdx.x < 32) {
    for (int j = threadIdx.x; j < n; j += 32) {
      s.x += q[j].x;
      s.y += q[j].y;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      s.x += __shfl_down_sync(0xffffffffu, s.x, o);
      s.y += __shfl_down_sync(0xffffffffu, s.y, o);
    }
  }
  return s;
}

// partial[v][m][blk] = sum over the block's slice of conj(a_m) * b
// a: nvec x ma vectors (stride lda per column, cols per vector = ma), b: one vector per vec.
template <class R>
__global__ void __launch_bounds__(kRedThreads)
k_dot_partial(const cx<R>* __restrict__ a, long long a_vstride, long long a_cstride, int ma,
              const cx<R>* __restrict__ b, long long b_vstride, long long len, double2* __restrict__ partial,
              const int* __restrict__ active) {
  const int vec = blockIdx.y;
  const int m = blockIdx.z;
  const int nblk = gridDim.x;
  double2* out = partial + ((long long)vec * ma + m) * nblk + blockIdx.x;
  pdl_wait();
  if (active && !active[vec]) {
    if (threadIdx.x == 0) *out = make_double2(0.0, 0.0);
    return;
  }
  const cx<R>* av = a + vec * a_vstride + m * a_cstride;
  const cx<R>* bv = b + vec * b_vstride;
  // Per-thread partial sums in the vector's own precision (a complex64 thread
  // sums a few dozen products; FP64 is rate-limited on this part), then FP64
  // across threads and blocks.
  R sx0 = 0, sy0 = 0, sx1 = 0, sy1 = 0;
  const long long chunk = (len + nblk - 1) / nblk, end = min(len, (blockIdx.x + 1) * chunk);
  long long i = blockIdx.x * chunk + threadIdx.x;
  for (; i + kRedThreads < end; i += 2 * kRedThreads) {
    cx<R> x = av[i], y = bv[i], x2 = av[i + kRedThreads], y2 = bv[i + kRedThreads];
    sx0 = rfma(x.x, y.x, rfma(x.y, y.y, sx0));
    sy0 = rfma(x.x, y.y, rfma(-x.y, y.x, sy0));
    sx1 = rfma(x2.x, y2.x, rfma(x2.y, y2.y, sx1));
    sy1 = rfma(x2.x, y2.y, rfma(-x2.y, y2.x, sy1));
  }
  if (i < end) {
    cx<R> x = av[i], y = bv[i];
    sx0 = rfma(x.x, y.x, rfma(x.y, y.y, sx0));
    sy0 = rfma(x.x, y.y, rfma(-x.y, y.x, sy0));
  }
  double2 s = make_double2(double(sx0) + double(sx1), double(sy0) + double(sy1));
  s = block_sum2(s);
  if (threadIdx.x == 0) *out = s;
}

// Residual update of the unpreconditioned CG: r -= a q ; partial (|r|^2, |r|^2).
template <class R>
__global__ void __launch_bounds__(kRedThreads)
k_cg_r_dot(cx<R>* __restrict__ r, const cx<R>* __restrict__ q, long long len, const double* __restrict__ alpha,
           const int* __restrict__ active, double2* __restrict__ partial) {
  const int vec = blockIdx.y;
  const int nblk = gridDim.x;
  double2* out = partial + (long long)vec * nblk + blockIdx.x;
  pdl_wait();
  if (active && !active[vec]) {
    if (threadIdx.x == 0) *out = make_double2(0.0, 0.0);
    return;
  }
  const R a = R(alpha[vec]);
  const long long o = vec * len;
  RunSum<R> s0;
  const long long chunk = (len + nblk - 1) / nblk, end = min(len, (blockIdx.x + 1) * chunk);
  for (long long i = blockIdx.x * chunk + threadIdx.x; i < end; i += kRedThreads) {
    const cx<R> ri = caxpy(-a, q[o + i], r[o + i]);
    r[o + i] = ri;
    s0.add(rfma(ri.x, ri.x, ri.y * ri.y));
  }
  const double2 s = block_sum2(make_double2(s0.value(), s0.value()));
  if (threadIdx.x == 0) *out = s;
}

__global__ void __launch_bounds__(32)
k_dot_final(const double2* __restrict__ partial, int nblk, double2* __restrict__ out) {
  const long long row = blockIdx.x;  // vec * ma + m
  pdl_wait();
  const double2 s = warp_sum2(partial + row * nblk, nblk);
  if (threadIdx.x == 0) out[row] = s;
}

// y_v = alpha_v * x_v + beta_v * y_v with per-vector complex scalars (FP64)
template <class R>
__global__ void k_axpby(const cx<R>* __restrict__ x, cx<R>* __restrict__ y, long long len, long long stride,
                        const double2* __restrict__ alpha, const double2* __restrict__ beta,
                        const int* __restrict__ active) {
  const int vec = blockIdx.y;
  if (active && !active[vec]) return;
  const double2 a = alpha[vec], bb = beta[vec];
  const cx<R>* xv = x + vec * stride;
  cx<R>* yv = y + vec * stride;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < len; i += (long long)gridDim.x * blockDim.x) {
    cx<R> xi = xv[i], yi = yv[i];
    double rx = a.x * xi.x - a.y * xi.y + bb.x * yi.x - bb.y * yi.y;
    double ry = a.x * xi.y + a.y * xi.x + bb.x * yi.y + bb.y * yi.x;
    yv[i] = mk<R>(R(rx), R(ry));
  }
}

__global__ void __launch_bounds__(32)
k_cg_alpha(const double2* __restrict__ partial, int nblk, double2* __restrict__ dot, const double* __restrict__ rho,
           double* __restrict__ alpha, int* __restrict__ active, int* __restrict__ iters, int* __restrict__ go) {
  const int v = blockIdx.x;
  pdl_wait();
  if (!active[v]) {
    if (threadIdx.x == 0) go[v] = 0;
    return;
  }
  const double2 s = warp_sum2(partial + (long long)v * nblk, nblk);
  if (threadIdx.x != 0) return;
  dot[v] = s;
  const bool ok = s.x > 0.0 && isfinite(s.x);
  alpha[v] = ok ? rho[v] / s.x : 0.0;
  go[v] = ok;
  if (!ok) {  // breakdown: B must be HPD
    active[v] = 0;
    iters[v] = -(iters[v] + 1);
  }
}

// Scalars of a CG solve from the partials (Re b^H z, |b|^2) of its start: rho,
// |b|^2, the stopping threshold (tol_v |b|)^2, the counts; vectors with a zero
// or non-finite right-hand side are not active.
__global__ void __launch_bounds__(32)
k_cg_init(const double2* __restrict__ partial, int nblk, const double* __restrict__ tolv, double* __restrict__ rho,
          double* __restrict__ tol2b2, double* __restrict__ bb, double* __restrict__ res2, int* __restrict__ active,
          int* __restrict__ iters) {
  const int v = blockIdx.x;
  pdl_wait();
  const double2 s = warp_sum2(partial + (long long)v * nblk, nblk);
  if (threadIdx.x != 0) return;
  rho[v] = s.x;
  bb[v] = s.y;
  res2[v] = s.y;
  tol2b2[v] = tolv[v] * tolv[v] * s.y;
  iters[v] = 0;
  if (!(s.y > 0.0) || !isfinite(s.y)) active[v] = 0;
}

// End of a CG iteration (cg_dir): x += alpha p, the convergence test, and p = z +
// beta p for the vectors that go on.  Every CTA of a vector reduces the partials
// in the same order, so all use the same beta; CTA 0 records the scalars.
// iters[v] counts the completed iterations of vector v on the device (so an
// iteration needs no host-side argument and can be replayed from a graph);
// a negative count flags breakdown at that iteration.
// HBM-bound (reads p, z, x, writes p and x: 141 MB in 24 us for 8 vectors at
// n = 48), the first elements loaded while the partials are reduced.  One launch
// replaces a scalar kernel (6 us of latency on one CTA per vector), the update
// of x in k_pcg_update (p is read once less: the two kernels 60 -> 53 us) and
// the one of p inside fncB's first plane kernel, which ran it at half the
// bandwidth.
// p and z are workspaces, x may be the caller's: with XALIGNED false (complex64
// at an odd element of a larger array) its elements are accessed one by one.
template <class R, bool XALIGNED>
__global__ void __launch_bounds__(kRedThreads)
k_cg_dir(cx<R>* __restrict__ x, cx<R>* __restrict__ p, const cx<R>* __restrict__ z, long long len,
         const double2* __restrict__ partial, int nblk, const double* __restrict__ alpha,
         const double* __restrict__ rho, double* __restrict__ rho_next, double2* __restrict__ dot,
         const double* __restrict__ tol2b2, const int* __restrict__ go, int* __restrict__ active,
         int* __restrict__ iters, double* __restrict__ res2) {
  const int v = blockIdx.y;
  __shared__ int s_act;
  __shared__ double s_beta;
  pdl_wait();
  // not active[v]: CTA 0 clears that one on convergence, and a CTA that starts
  // after it still owes its part of x
  if (!go[v]) return;
  constexpr int U = 16 / sizeof(cx<R>);  // elements per 16-byte access (len is a multiple of 4)
  struct alignas(16) Pack {
    cx<R> e[U];
  };
  cx<R>* xv = x + (long long)v * len;
  Pack* pp = reinterpret_cast<Pack*>(p + (long long)v * len);
  const Pack* zp = reinterpret_cast<const Pack*>(z + (long long)v * len);
  const int np = int(len / U), chunk = (np + gridDim.x - 1) / gridDim.x;
  const int end = min(np, (int(blockIdx.x) + 1) * chunk);
  int i = blockIdx.x * chunk + threadIdx.x;
  constexpr int B = 3;  // packs of each in flight; the first ones during the reduction
  Pack a[B], c[B], e[B];
  auto load = [&]() {
#pragma unroll
    for (int u = 0; u < B; ++u)
      if (i + u * kRedThreads < end) {
        a[u] = zp[i + u * kRedThreads];
        c[u] = pp[i + u * kRedThreads];
        cx<R>* xe = xv + (long long)(i + u * kRedThreads) * U;
        if constexpr (XALIGNED) {
          e[u] = *reinterpret_cast<const Pack*>(xe);
        } else {
#pragma unroll
          for (int w = 0; w < U; ++w) e[u].e[w] = xe[w];
        }
      }
  };
  load();
  const double2 s = warp_sum2(partial + (long long)v * nblk, nblk);
  if (threadIdx.x == 0) {
    const double rz = s.x, rn = s.y;  // (Re r'z, |r|^2), z = M r (z = r without preconditioner)
    const double r0 = rho[v];
    s_beta = r0 != 0.0 ? rz / r0 : 0.0;
    const bool bad = !isfinite(rn) || !isfinite(rz);
    const bool conv = !bad && rn <= tol2b2[v];        // ||r|| <= tol ||b||
    const bool indef = !bad && !conv && !(rz > 0.0);  // indefinite preconditioned system
    s_act = !(bad || conv || indef);
    if (blockIdx.x == 0) {
      const int it = iters[v] + 1;
      dot[v] = s;
      res2[v] = rn;
      rho_next[v] = rz;
      iters[v] = bad || indef ? -it : it;
      if (!s_act) active[v] = 0;
    }
  }
  __syncthreads();
  const bool more = s_act != 0;  // a vector that stops here needs no further direction
  const R al = R(alpha[v]), b = R(s_beta);
  while (i < end) {
#pragma unroll
    for (int u = 0; u < B; ++u)
      if (i + u * kRedThreads < end) {
#pragma unroll
        for (int w = 0; w < U; ++w) {
          e[u].e[w] = caxpy(al, c[u].e[w], e[u].e[w]);
          c[u].e[w] = caxpy(b, c[u].e[w], a[u].e[w]);
        }
        cx<R>* xe = xv + (long long)(i + u * kRedThreads) * U;
        if constexpr (XALIGNED) {
          *reinterpret_cast<Pack*>(xe) = e[u];
        } else {
#pragma unroll
          for (int w = 0; w < U; ++w) xe[w] = e[u].e[w];
        }
        if (more) pp[i + u * kRedThreads] = c[u];
      }
    i += B * kRedThreads;
    load();
  }
}

// out[:, j] = sum_i in[:, i] * U[i, j]  (U real, p x k, column-major), all columns of one vector block
template <class R>
__global__ void k_block_rot(const cx<R>* __restrict__ in, cx<R>* __restrict__ out, long long len,
                            long long ld, int p, int k, const double* __restrict__ U) {
  extern __shared__ double Us[];
  for (int i = threadIdx.x; i < p * k; i += blockDim.x) Us[i] = U[i];
  __syncthreads();
  for (long long row = (long long)blockIdx.x * blockDim.x + threadIdx.x; row < len; row += (long long)gridDim.x * blockDim.x) {
    for (int j = 0; j < k; ++j) {
      double sx = 0.0, sy = 0.0;
      for (int i = 0; i < p; ++i) {
        cx<R> q = in[(long long)i * ld + row];
        sx += double(q.x) * Us[j * p + i];
        sy += double(q.y) * Us[j * p + i];
      }
      out[(long long)j * ld + row] = mk<R>(R(sx), R(sy));
    }
  }
}

// out = a x + b y + c w (real scalars; y, w may be null)
template <class R>
__global__ void k_lincomb3(cx<R>* out, double a, const cx<R>* x, double b, const cx<R>* y, double c, const cx<R>* w,
                           long long len) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < len; i += (long long)gridDim.x * blockDim.x) {
    cx<R> xi = x[i];
    double rx = a * xi.x, ry = a * xi.y;
    if (y) {
      cx<R> yi = y[i];
      rx += b * yi.x;
      ry += b * yi.y;
    }
    if (w) {
      cx<R> wi = w[i];
      rx += c * wi.x;
      ry += c * wi.y;
    }
    out[i] = mk<R>(R(rx), R(ry));
  }
}

// out[:, j] = sum_i in[:, i] * C[i, j]  (C complex m x q, column-major)
template <class R>
__global__ void k_block_comb(const cx<R>* __restrict__ in, cx<R>* __restrict__ out, long long len, long long ld,
                             int m, int q, const double2* __restrict__ C) {
  extern __shared__ double2 Cs[];
  for (int i = threadIdx.x; i < m * q; i += blockDim.x) Cs[i] = C[i];
  __syncthreads();
  for (long long row = (long long)blockIdx.x * blockDim.x + threadIdx.x; row < len; row += (long long)gridDim.x * blockDim.x) {
    for (int j = 0; j < q; ++j) {
      double sx = 0.0, sy = 0.0;
      for (int i = 0; i < m; ++i) {
        const cx<R> v = in[(long long)i * ld + row];
        const double2 c = Cs[j * m + i];
        sx += double(v.x) * c.x - double(v.y) * c.y;
        sy += double(v.x) * c.y + double(v.y) * c.x;
      }
      out[(long long)j * ld + row] = mk<R>(R(sx), R(sy));
    }
  }
}

// ---------------------------------------------------------------------------
// Gram-Schmidt over a batch of k-point instances in one launch each: vector v
// works against its own columns col0_v .. col0_v + m_v - 1 (span[v] = (col0, m),
// m = 0 skips it) of its block X + v * xs (columns len apart).
// ---------------------------------------------------------------------------
// partial[(v * maxm + i) * nblk + blk] = block's share of X_v[col0_v + i]^H r_v
// FP64-rate-bound (4 fused operations per element; 12 -> 7 us a column of 4 x
// 256000 with them, where the plain expressions take 6).
__global__ void __launch_bounds__(kRedThreads)
k_gs_dot_partial(const double2* __restrict__ X, long long xs, const double2* __restrict__ r, long long rs,
                 long long len, const int2* __restrict__ span, int maxm, double2* __restrict__ partial) {
  const int v = blockIdx.y, i = blockIdx.z, nblk = gridDim.x;
  pdl_wait();
  const int2 sp = span[v];
  if (i >= sp.y) return;
  const double2* a = X + v * xs + (long long)(sp.x + i) * len;
  const double2* b = r + v * rs;
  double sx0 = 0.0, sy0 = 0.0, sx1 = 0.0, sy1 = 0.0;
  const long long chunk = (len + nblk - 1) / nblk, end = min(len, (blockIdx.x + 1) * chunk);
  long long k = blockIdx.x * chunk + threadIdx.x;
  for (; k + kRedThreads < end; k += 2 * kRedThreads) {
    const double2 x = a[k], y = b[k], x2 = a[k + kRedThreads], y2 = b[k + kRedThreads];
    sx0 = rfma(x.x, y.x, rfma(x.y, y.y, sx0));
    sy0 = rfma(x.x, y.y, rfma(-x.y, y.x, sy0));
    sx1 = rfma(x2.x, y2.x, rfma(x2.y, y2.y, sx1));
    sy1 = rfma(x2.x, y2.y, rfma(-x2.y, y2.x, sy1));
  }
  if (k < end) {
    const double2 x = a[k], y = b[k];
    sx0 = rfma(x.x, y.x, rfma(x.y, y.y, sx0));
    sy0 = rfma(x.x, y.y, rfma(-x.y, y.x, sy0));
  }
  const double2 s = block_sum2(make_double2(sx0 + sx1, sy0 + sy1));
  if (threadIdx.x == 0) partial[((long long)v * maxm + i) * nblk + blockIdx.x] = s;
}

// coef[v * cstride + i] = sum over blocks (i < m_v)
__global__ void __launch_bounds__(32)
k_gs_dot_final(const double2* __restrict__ partial, int nblk, int maxm, const int2* __restrict__ span,
               double2* __restrict__ coef, int cstride) {
  const int v = blockIdx.x / maxm, i = blockIdx.x - v * maxm;
  pdl_wait();
  if (i >= span[v].y) return;
  const double2 s = warp_sum2(partial + ((long long)v * maxm + i) * nblk, nblk);
  if (threadIdx.x == 0) coef[(long long)v * cstride + i] = s;
}

// r_v -= sum_i coef[v * cstride + i] X_v[col0_v + i], and with r2 the same with X2
// (blockIdx.z), FP64 or from complex64 copies (the correction in FP32).  FP64:
// rate-bound, 4 fused operations per column and row.  complex64: HBM-bound; the
// coefficients are rounded once per CTA (converting them at every use kept the
// FP64 pipe busy for 31 of 44 us at 9 columns of 4 x 256000), 16-byte loads.
template <class XT>
__global__ void __launch_bounds__(kRedThreads)
k_gs_combo(double2* __restrict__ r, double2* __restrict__ r2, long long rs, const XT* __restrict__ X,
           const XT* __restrict__ X2, long long xs, long long len, const int2* __restrict__ span,
           const double2* __restrict__ coef, int cstride) {
  using S = decltype(XT::x);
  constexpr int U = 16 / sizeof(XT);  // rows per access (len is a multiple of 4)
  struct alignas(16) Pack {
    XT e[U];
  };
  __shared__ XT cs[128];
  const int v = blockIdx.y;
  pdl_wait();
  const int2 sp = span[v];
  if (sp.y <= 0) return;
  for (int i = threadIdx.x; i < sp.y; i += kRedThreads) {
    const double2 c = coef[(long long)v * cstride + i];
    cs[i] = mk<S>(S(c.x), S(c.y));
  }
  const int np = int(len / U);
  const Pack* x = reinterpret_cast<const Pack*>((blockIdx.z ? X2 : X) + v * xs + (long long)sp.x * len);
  double2* rv = (blockIdx.z ? r2 : r) + v * rs;
  __syncthreads();
  for (int k = blockIdx.x * kRedThreads + threadIdx.x; k < np; k += gridDim.x * kRedThreads) {
    XT acc[U];
#pragma unroll
    for (int u = 0; u < U; ++u) acc[u] = mk<S>(S(0), S(0));
    double2 o[U];
#pragma unroll
    for (int u = 0; u < U; ++u) o[u] = rv[(long long)k * U + u];
    int i = 0;
    for (; i + 4 <= sp.y; i += 4) {  // four columns' loads in flight
      Pack q[4];
#pragma unroll
      for (int w = 0; w < 4; ++w) q[w] = x[(long long)(i + w) * np + k];
#pragma unroll
      for (int w = 0; w < 4; ++w)
#pragma unroll
        for (int u = 0; u < U; ++u) acc[u] = cfma(cs[i + w], q[w].e[u], acc[u]);
    }
    for (; i < sp.y; ++i) {
      const Pack q = x[(long long)i * np + k];
#pragma unroll
      for (int u = 0; u < U; ++u) acc[u] = cfma(cs[i], q.e[u], acc[u]);
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      o[u].x -= double(acc[u].x);
      o[u].y -= double(acc[u].y);
      rv[(long long)k * U + u] = o[u];
    }
  }
}

// r -= sum_i c_i X[:, i]  (complex coefficients, FP64)
template <class R>
__global__ void k_sub_combo(cx<R>* __restrict__ r, const cx<R>* __restrict__ X, long long len, long long ld, int m,
                            const double2* __restrict__ c) {
  extern __shared__ double2 cs[];
  for (int i = threadIdx.x; i < m; i += blockDim.x) cs[i] = c[i];
  __syncthreads();
  for (long long row = (long long)blockIdx.x * blockDim.x + threadIdx.x; row < len; row += (long long)gridDim.x * blockDim.x) {
    cx<R> acc = r[row];
    double ax = acc.x, ay = acc.y;
    for (int i = 0; i < m; ++i) {
      cx<R> q = X[(long long)i * ld + row];
      ax -= cs[i].x * q.x - cs[i].y * q.y;
      ay -= cs[i].x * q.y + cs[i].y * q.x;
    }
    r[row] = mk<R>(R(ax), R(ay));
  }
}

template <class D, class S>
__global__ void k_convert(const cx<S>* __restrict__ in, cx<D>* __restrict__ out, long long n) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    out[i] = mk<D>(D(in[i].x), D(in[i].y));
}

// x64 += m_v * d32 (m null: m_v = 1); res = b - bx (both FP64) for active vectors
__global__ void k_refine_acc(double2* __restrict__ x, const float2* __restrict__ d, long long len,
                             const int* __restrict__ active, const double* __restrict__ mult) {
  const int vec = blockIdx.y;
  if (active && !active[vec]) return;
  const double m = mult ? mult[vec] : 1.0;
  const long long o = vec * len;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < len; i += (long long)gridDim.x * blockDim.x) {
    double2 a = x[o + i];
    float2 b = d[o + i];
    a.x += m * double(b.x);
    a.y += m * double(b.y);
    x[o + i] = a;
  }
}
__global__ void k_residual(const double2* __restrict__ b, const double2* __restrict__ bx, double2* __restrict__ res,
                           float2* __restrict__ res32, long long len, const int* __restrict__ active) {
  const int vec = blockIdx.y;
  if (active && !active[vec]) return;
  const long long o = vec * len;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < len; i += (long long)gridDim.x * blockDim.x) {
    double2 r = make_double2(b[o + i].x - bx[o + i].x, b[o + i].y - bx[o + i].y);
    res[o + i] = r;
    if (res32) res32[o + i] = make_float2(float(r.x), float(r.y));
  }
}
// out32 = s_v * in (FP64 -> complex64) for active vectors
__global__ void k_to32_scaled(const double2* __restrict__ in, float2* __restrict__ out, long long len,
                              const double* __restrict__ s, const int* __restrict__ active) {
  const int vec = blockIdx.y;
  if (active && !active[vec]) return;
  const double a = s[vec];
  const long long o = vec * len;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < len; i += (long long)gridDim.x * blockDim.x) {
    const double2 r = in[o + i];
    out[o + i] = make_float2(float(a * r.x), float(a * r.y));
  }
}
// y = s_v * x per vector (real per-vector scalars), x and y may alias
template <class R>
__global__ void k_scale(const cx<R>* x, cx<R>* y, long long len, const double* __restrict__ s,
                        const int* __restrict__ active) {
  const int vec = blockIdx.y;
  if (active && !active[vec]) return;
  const R a = R(s[vec]);
  const long long o = vec * len;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < len; i += (long long)gridDim.x * blockDim.x) {
    cx<R> v = x[o + i];
    y[o + i] = mk<R>(a * v.x, a * v.y);
  }
}

int grid_for(long long len) {
  long long b = (len + 255) / 256;
  if (b > 4096) b = 4096;
  return int(b < 1 ? 1 : b);
}

}  // namespace

template <class R>
cudaError_t dot_batched(const cx<R>* a, long long a_vstride, long long a_cstride, int ma, const cx<R>* b,
                        long long b_vstride, long long len, int nvec, double2* out, double2* partial,
                        int nblk, const int* active, cudaStream_t st) {
  if (nvec <= 0 || ma <= 0) return cudaSuccess;
  cudaError_t e = launch<k_dot_partial<R>>(dim3(nblk, nvec, ma), kRedThreads, 0, st, a, a_vstride, a_cstride, ma, b,
                                               b_vstride, len, partial, active);
  if (e != cudaSuccess) return e;
  return launch<k_dot_final>(dim3(nvec * ma), 32, 0, st, (const double2*)partial, nblk, out);
}

template <class R>
cudaError_t axpby_batched(const cx<R>* x, cx<R>* y, long long len, long long stride, int nvec,
                          const double2* alpha, const double2* beta, const int* active, cudaStream_t st) {
  if (nvec <= 0) return cudaSuccess;
  int gx = grid_for(len);
  if (gx > 1024) gx = 1024;
  FAME_LAUNCHED(1);
  k_axpby<R><<<dim3(gx, nvec), 256, 0, st>>>(x, y, len, stride, alpha, beta, active);
  return cudaGetLastError();
}

template <class R>
cudaError_t dot_partial(const cx<R>* a, const cx<R>* b, long long len, long long stride, int nvec, double2* partial,
                        int nblk, const int* active, cudaStream_t st) {
  if (nvec <= 0) return cudaSuccess;
  return launch<k_dot_partial<R>>(dim3(nblk, nvec, 1), kRedThreads, 0, st, a, stride, 0LL, 1, b, stride, len, partial,
                                      active);
}

template <class R>
cudaError_t cg_r_partial(cx<R>* r, const cx<R>* q, long long len, int nvec, const double* alpha, const int* active,
                         double2* partial, int nblk, cudaStream_t st) {
  return launch<k_cg_r_dot<R>>(dim3(nblk, nvec), kRedThreads, 0, st, r, q, len, alpha, active, partial);
}

// Q_v[:, col_v] = V_v, BQ_v[:, col_v] = BV_v (and their complex64 copies when
// given) for every v with col_v >= 0.
__global__ void k_gs_store(double2* __restrict__ Q, double2* __restrict__ BQ, float2* __restrict__ Q32,
                           float2* __restrict__ BQ32, long long xs, const double2* __restrict__ V,
                           const double2* __restrict__ BV, long long len, const int* __restrict__ col) {
  const int v = blockIdx.y;
  const int c = col[v];
  if (c < 0) return;
  const long long o = v * xs + (long long)c * len;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < len; i += (long long)gridDim.x * blockDim.x) {
    const double2 a = V[v * len + i], b = BV[v * len + i];
    Q[o + i] = a;
    BQ[o + i] = b;
    if (Q32) {
      Q32[o + i] = make_float2(float(a.x), float(a.y));
      BQ32[o + i] = make_float2(float(b.x), float(b.y));
    }
  }
}

cudaError_t gs_store(double2* Q, double2* BQ, float2* Q32, float2* BQ32, long long xs, const double2* V,
                     const double2* BV, long long len, int nv, const int* col, cudaStream_t st) {
  if (nv <= 0) return cudaSuccess;
  int gx = grid_for(len);
  if (gx > 1024) gx = 1024;
  FAME_LAUNCHED(1);
  k_gs_store<<<dim3(gx, nv), 256, 0, st>>>(Q, BQ, Q32, BQ32, xs, V, BV, len, col);
  return cudaGetLastError();
}

cudaError_t gs_dots(const double2* X, long long xs, const double2* r, long long rs, long long len, int nv,
                    const int2* span, int maxm, double2* coef, int cstride, double2* partial, int nblk,
                    cudaStream_t st) {
  if (nv <= 0 || maxm <= 0) return cudaSuccess;
  cudaError_t e = launch<k_gs_dot_partial>(dim3(nblk, nv, maxm), kRedThreads, 0, st, X, xs, r, rs, len, span, maxm,
                                           partial);
  if (e != cudaSuccess) return e;
  return launch<k_gs_dot_final>(dim3(nv * maxm), 32, 0, st, (const double2*)partial, nblk, maxm, span, coef, cstride);
}

template <class XT>
cudaError_t gs_combo(double2* r, double2* r2, long long rs, const XT* X, const XT* X2, long long xs, long long len,
                     int nv, const int2* span, const double2* coef, int cstride, cudaStream_t st) {
  if (nv <= 0) return cudaSuccess;
  const int gx = (int)std::min(1024LL, (len * (long long)sizeof(XT) / 16 + kRedThreads - 1) / kRedThreads);
  return launch<k_gs_combo<XT>>(dim3(gx, nv, r2 ? 2 : 1), kRedThreads, 0, st, r, r2, rs, X, X2, xs, len, span, coef,
                                cstride);
}
template cudaError_t gs_combo<double2>(double2*, double2*, long long, const double2*, const double2*, long long,
                                       long long, int, const int2*, const double2*, int, cudaStream_t);
template cudaError_t gs_combo<float2>(double2*, double2*, long long, const float2*, const float2*, long long,
                                      long long, int, const int2*, const double2*, int, cudaStream_t);

// The loop condition of a graph-resident iteration loop: one pass of the
// body done (*passes + 1); continue while any vector is active and fewer
// than max_passes passes have run.
__global__ void k_while_active(const int* __restrict__ active, int nvec, int* __restrict__ passes, int max_passes,
                               cudaGraphConditionalHandle h) {
  int any = 0;
  for (int v = threadIdx.x; v < nvec; v += blockDim.x) any |= active[v];
  any = __any_sync(0xffffffffu, any);
  if (threadIdx.x == 0) {
    const int b = *passes + 1;
    *passes = b;
    cudaGraphSetConditional(h, (any && b < max_passes) ? 1u : 0u);
  }
}

cudaError_t while_active(const int* active, int nvec, int* passes, int max_passes, cudaGraphConditionalHandle h,
                         cudaStream_t st) {
  FAME_LAUNCHED(1);
  k_while_active<<<1, 32, 0, st>>>(active, nvec, passes, max_passes, h);
  return cudaGetLastError();
}

cudaError_t cg_alpha(int nvec, const double2* partial, int nblk, double2* dot, const double* rho, double* alpha,
                     int* active, int* iters, int* go, cudaStream_t st) {
  return launch<k_cg_alpha>(dim3(nvec), 32, 0, st, partial, nblk, dot, rho, alpha, active, iters, go);
}

cudaError_t cg_init(int nvec, const double2* partial, int nblk, const double* tolv, double* rho, double* tol2b2,
                    double* bb, double* res2, int* active, int* iters, cudaStream_t st) {
  return launch<k_cg_init>(dim3(nvec), 32, 0, st, partial, nblk, tolv, rho, tol2b2, bb, res2, active, iters);
}

template <class R>
cudaError_t cg_dir(cx<R>* x, cx<R>* p, const cx<R>* z, long long len, int nvec, const double2* partial, int nblk,
                   const double* alpha, const double* rho, double* rho_next, double2* dot, const double* tol2b2,
                   const int* go, int* active, int* iters, double* res2, int ncta, cudaStream_t st) {
  if constexpr (sizeof(cx<R>) < 16)
    if ((uintptr_t)x % 16 != 0)  // every vector then, as len is even
      return launch<k_cg_dir<R, false>>(dim3(ncta, nvec), kRedThreads, 0, st, x, p, z, len, partial, nblk, alpha, rho,
                                        rho_next, dot, tol2b2, go, active, iters, res2);
  return launch<k_cg_dir<R, true>>(dim3(ncta, nvec), kRedThreads, 0, st, x, p, z, len, partial, nblk, alpha, rho, rho_next,
                                   dot, tol2b2, go, active, iters, res2);
}

template <class R>
cudaError_t block_rot(const cx<R>* in, cx<R>* out, long long len, long long ld, int p, int k, const double* U,
                      cudaStream_t st) {
  FAME_LAUNCHED(1);
  k_block_rot<R><<<grid_for(len), 256, sizeof(double) * p * k, st>>>(in, out, len, ld, p, k, U);
  return cudaGetLastError();
}

template <class R>
cudaError_t lincomb3(cx<R>* out, double a, const cx<R>* x, double b, const cx<R>* y, double c, const cx<R>* w,
                     long long len, cudaStream_t st) {
  FAME_LAUNCHED(1);
  k_lincomb3<R><<<grid_for(len), 256, 0, st>>>(out, a, x, b, y, c, w, len);
  return cudaGetLastError();
}
template cudaError_t lincomb3<float>(cx<float>*, double, const cx<float>*, double, const cx<float>*, double,
                                     const cx<float>*, long long, cudaStream_t);
template cudaError_t lincomb3<double>(cx<double>*, double, const cx<double>*, double, const cx<double>*, double,
                                      const cx<double>*, long long, cudaStream_t);

template <class R>
cudaError_t block_comb(const cx<R>* in, cx<R>* out, long long len, long long ld, int m, int q, const double2* C,
                       cudaStream_t st) {
  const size_t sm = sizeof(double2) * m * q;
  if (sm > 200 * 1024) return cudaErrorInvalidValue;
  if (sm > 48 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(k_block_comb<R>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    if (e != cudaSuccess) return e;
  }
  FAME_LAUNCHED(1);
  k_block_comb<R><<<grid_for(len), 256, sm, st>>>(in, out, len, ld, m, q, C);
  return cudaGetLastError();
}
template cudaError_t block_comb<double>(const cx<double>*, cx<double>*, long long, long long, int, int, const double2*,
                                        cudaStream_t);

template <class R>
cudaError_t sub_combo(cx<R>* r, const cx<R>* X, long long len, long long ld, int m, const double2* c,
                      cudaStream_t st) {
  if (m <= 0) return cudaSuccess;
  FAME_LAUNCHED(1);
  k_sub_combo<R><<<grid_for(len), 256, sizeof(double2) * m, st>>>(r, X, len, ld, m, c);
  return cudaGetLastError();
}

template <class D, class S>
cudaError_t convert(const cx<S>* in, cx<D>* out, long long n, cudaStream_t st) {
  FAME_LAUNCHED(1);
  k_convert<D, S><<<grid_for(n), 256, 0, st>>>(in, out, n);
  return cudaGetLastError();
}

cudaError_t refine_acc(double2* x, const float2* d, long long len, int nvec, const int* active, cudaStream_t st,
                       const double* mult) {
  int gx = grid_for(len);
  if (gx > 1024) gx = 1024;
  FAME_LAUNCHED(1);
  k_refine_acc<<<dim3(gx, nvec), 256, 0, st>>>(x, d, len, active, mult);
  return cudaGetLastError();
}

cudaError_t to32_scaled(const double2* in, float2* out, long long len, int nvec, const double* s, const int* active,
                        cudaStream_t st) {
  int gx = grid_for(len);
  if (gx > 1024) gx = 1024;
  FAME_LAUNCHED(1);
  k_to32_scaled<<<dim3(gx, nvec), 256, 0, st>>>(in, out, len, s, active);
  return cudaGetLastError();
}

cudaError_t residual(const double2* b, const double2* bx, double2* res, float2* res32, long long len, int nvec,
                     const int* active, cudaStream_t st) {
  int gx = grid_for(len);
  if (gx > 1024) gx = 1024;
  FAME_LAUNCHED(1);
  k_residual<<<dim3(gx, nvec), 256, 0, st>>>(b, bx, res, res32, len, active);
  return cudaGetLastError();
}

template <class R>
cudaError_t scale_batched(const cx<R>* x, cx<R>* y, long long len, int nvec, const double* s, const int* active,
                          cudaStream_t st) {
  int gx = grid_for(len);
  if (gx > 1024) gx = 1024;
  FAME_LAUNCHED(1);
  k_scale<R><<<dim3(gx, nvec), 256, 0, st>>>(x, y, len, s, active);
  return cudaGetLastError();
}
template cudaError_t scale_batched<double>(const cx<double>*, cx<double>*, long long, int, const double*, const int*,
                                           cudaStream_t);
template cudaError_t scale_batched<float>(const cx<float>*, cx<float>*, long long, int, const double*, const int*,
                                          cudaStream_t);

#define FAME_KINST(R)                                                                                     \
  template cudaError_t dot_batched<R>(const cx<R>*, long long, long long, int, const cx<R>*, long long,  \
                                      long long, int, double2*, double2*, int, const int*, cudaStream_t); \
  template cudaError_t axpby_batched<R>(const cx<R>*, cx<R>*, long long, long long, int, const double2*, \
                                        const double2*, const int*, cudaStream_t);                       \
  template cudaError_t cg_dir<R>(cx<R>*, cx<R>*, const cx<R>*, long long, int, const double2*, int,        \
                                 const double*, const double*, double*, double2*, const double*,          \
                                 const int*, int*, int*, double*, int, cudaStream_t);                     \
  template cudaError_t block_rot<R>(const cx<R>*, cx<R>*, long long, long long, int, int, const double*, \
                                    cudaStream_t);                                                        \
  template cudaError_t sub_combo<R>(cx<R>*, const cx<R>*, long long, long long, int, const double2*,     \
                                    cudaStream_t);                                                        \
  template cudaError_t dot_partial<R>(const cx<R>*, const cx<R>*, long long, long long, int, double2*,   \
                                      int, const int*, cudaStream_t);                                     \
  template cudaError_t cg_r_partial<R>(cx<R>*, const cx<R>*, long long, int, const double*, const int*,     \
                                       double2*, int, cudaStream_t);
FAME_KINST(float)
FAME_KINST(double)
template cudaError_t convert<float, double>(const cx<double>*, cx<float>*, long long, cudaStream_t);
template cudaError_t convert<double, float>(const cx<float>*, cx<double>*, long long, cudaStream_t);

}  // namespace fame

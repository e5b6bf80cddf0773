// The FP64 side of the batched BiCGStab, for every right-hand side of a block in one
// launch per step: the first residual, and the reliable updates of the right-hand sides
// that went pending.  Each kernel runs over (sites, right-hand side) and a block whose
// right-hand side is not concerned leaves at once, so an update costs six launches however
// many right-hand sides take part, and the lattice of one right-hand side need not fill
// the GPU by itself.  (One right-hand side at a time, twelve launches each: twelve point
// sources on 8^3x16 at kappa = 0.150 took 21.4 ms, now 11.1; on 24^3x48 twisted 330 ms,
// now 302.)  The kernels stream FP64 fields; slot k of a block field is read 16 bytes in
// every 16 nb, half of each sector.
#include <cmath>

#include "qq_pend.h"

namespace qq {
namespace {

constexpr int kPendThreads = 128;

__device__ inline bool pend_on(const unsigned* ctl, int mask, int k) {
  const unsigned w = mask == PEND_ALL ? 0xffffffffu
                     : mask == PEND_PENDING ? ctl[CTL_PENDING] & ~ctl[CTL_DONE] : ctl[CTL_INSERT];
  return (w >> k) & 1u;
}

// x += xl, xl = 0 for the pending right-hand sides.
template <int P>
__global__ void __launch_bounds__(kPendThreads) pend_accum_kernel(PendArgs A) {
  const int k = blockIdx.y;
  if (!pend_on(A.ctl, PEND_PENDING, k)) return;
  const int s = blockIdx.x * kPendThreads + threadIdx.x;
  if (s >= A.vh) return;
  using RB = typename SpinorIO<P>::R;
  const int e = s * A.nb + k, n = A.vh * A.nb;
  void* x = static_cast<char*>(A.x) + A.stride * A.rhs[k];
  cplx<RB> b[12];
  cplx<double> v[12];
  SpinorIO<P64>::load(x, nullptr, A.vh, s, v);
  SpinorIO<P>::load(A.xl.data, A.xl.norm, n, e, b);
#pragma unroll
  for (int q = 0; q < 12; ++q) {
    v[q] = {v[q].re + (double)b[q].re, v[q].im + (double)b[q].im};
    b[q] = {(RB)0, (RB)0};
  }
  SpinorIO<P64>::store(x, nullptr, A.vh, s, v);
  SpinorIO<P>::store(A.xl.data, A.xl.norm, n, e, b);
}

// First (RES = 0) and second (RES = 1) hop of r = b - A x; the second also sums ||r||^2
// and, when A.norm_b is set, ||b||^2.  EPI: EPI_STORE or EPI_TWIST of the first hop.
template <int RECON, int EPI, int RES>
__global__ void __launch_bounds__(kPendThreads, 3) pend_hop_kernel(HopArgs h, PendArgs A, int mask) {
  const int k = blockIdx.y;
  if (!pend_on(A.ctl, mask, k)) return;
  const int s = blockIdx.x * kPendThreads + threadIdx.x;
  const size_t mine = A.stride * k, off = A.stride * A.rhs[k];
  h.in[0] = RES ? static_cast<const char*>(A.tmp) + mine : static_cast<const char*>(A.x) + off;
  h.out[0] = static_cast<char*>(RES ? A.r64 : A.tmp) + mine;
  double n2 = 0.0, b2 = 0.0;
  if (s < A.vh) {
    int x[4];
    site_coords(h.g, h.pout, s, x);
    cplx<double> acc[12];
#pragma unroll
    for (int c = 0; c < 12; ++c) acc[c] = {0.0, 0.0};
    hop<P64, P64, RECON, 0, true>(h, s, 0, x, acc);
    hop<P64, P64, RECON, 0, false>(h, s, 0, x, acc);
    hop<P64, P64, RECON, 1, true>(h, s, 0, x, acc);
    hop<P64, P64, RECON, 1, false>(h, s, 0, x, acc);
    hop<P64, P64, RECON, 2, true>(h, s, 0, x, acc);
    hop<P64, P64, RECON, 2, false>(h, s, 0, x, acc);
    hop<P64, P64, RECON, 3, true>(h, s, 0, x, acc);
    hop<P64, P64, RECON, 3, false>(h, s, 0, x, acc);
    if (RES == 0) {
      hop_finish<P64, EPI>(h, s, 0, acc);
    } else {
      cplx<double> g[12], b[12];
      SpinorIO<P64>::load(static_cast<const char*>(A.x) + off, nullptr, A.vh, s, g);
      SpinorIO<P64>::load(static_cast<const char*>(A.b) + off, nullptr, A.vh, s, b);
#pragma unroll
      for (int c = 0; c < 6; ++c) {
        // A x = f1 x + f2 J x - f3 H tmp, J(v) = (v2, v3, -v0, -v1)
        const cplx<double> up = csub(cadd(cscale(h.f1, g[c]), cscale(h.f2, g[6 + c])), cscale(h.f3, acc[c]));
        const cplx<double> lo = csub(csub(cscale(h.f1, g[6 + c]), cscale(h.f2, g[c])), cscale(h.f3, acc[6 + c]));
        acc[c] = csub(b[c], up);
        acc[6 + c] = csub(b[6 + c], lo);
      }
#pragma unroll
      for (int c = 0; c < 12; ++c) {
        n2 += acc[c].re * acc[c].re + acc[c].im * acc[c].im;
        b2 += b[c].re * b[c].re + b[c].im * b[c].im;
      }
      SpinorIO<P64>::store(h.out[0], nullptr, A.vh, s, acc);
    }
  }
  if (RES == 0) return;
  __shared__ double red[2][kPendThreads / 32];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    n2 += __shfl_down_sync(0xffffffffu, n2, o);
    b2 += __shfl_down_sync(0xffffffffu, b2, o);
  }
  if ((threadIdx.x & 31) == 0) {
    red[0][threadIdx.x >> 5] = n2;
    red[1][threadIdx.x >> 5] = b2;
  }
  __syncthreads();
  if (threadIdx.x < 2) {
    double t = 0.0;
    for (int w = 0; w < kPendThreads / 32; ++w) t += red[threadIdx.x][w];
    A.partial[((size_t)k * 2 + threadIdx.x) * gridDim.x + blockIdx.x] = t;
  }
}

// Sum of n values in a fixed order by a block of 256 threads (the same in every thread).
__device__ inline double pend_sum(const double* v, int n) {
  __shared__ double red[256];
  double s = 0.0;
  for (int b = threadIdx.x; b < n; b += 256) s += v[b];
  __syncthreads();
  red[threadIdx.x] = s;
  __syncthreads();
  for (int o = 128; o > 0; o >>= 1) {
    if (threadIdx.x < o) red[threadIdx.x] += red[threadIdx.x + o];
    __syncthreads();
  }
  return red[0];
}

// The scalars of right-hand side blockIdx.x before its first iteration: rhat = r = the
// FP64 residual of the initial guess, whose norm also anchors the stall test, so rho =
// <rhat, r> = ||r||^2; with p = v = 0 the first search direction is r whatever beta is.
__global__ void __launch_bounds__(256) pend_init_kernel(PendArgs A, int nblocks) {
  const int k = blockIdx.x;
  const double r2 = pend_sum(A.partial + (size_t)k * 2 * nblocks, nblocks);
  const double b2 = pend_sum(A.partial + ((size_t)k * 2 + 1) * nblocks, nblocks);
  if (threadIdx.x != 0) return;
  double* s = A.S + (size_t)k * kScal;
  for (int q = 0; q < kScal; ++q) s[q] = 0.0;
  const double rn = sqrt(r2), bn = sqrt(b2);
  s[SC_ALPHA] = s[SC_OMEGA] = 1.0;
  s[SC_RHO] = rn * rn;
  s[SC_RMAX] = rn;
  s[SC_BN] = bn > 0.0 ? bn : 1.0;
  s[SC_R2] = rn * rn;
  s[SC_RHATN] = rn;
  s[SC_CHK_R] = rn;
  s[SC_TRUE] = bn > 0.0 ? rn / bn : 0.0;
  s[SC_T2] = b2;
  atomicOr(&A.ctl[!(bn > 0.0) || rn / bn <= A.tol ? CTL_DONE : CTL_ACTIVE], 1u << k);
}

// The decision of right-hand side blockIdx.x's reliable update.
__global__ void __launch_bounds__(256) pend_decide_kernel(PendArgs A, int nblocks) {
  const int k = blockIdx.x;
  const bool on = pend_on(A.ctl, PEND_PENDING, k);
  __syncthreads();  // every thread has read the mask that thread 0 changes below
  if (!on) return;
  const double r2 = pend_sum(A.partial + (size_t)k * 2 * nblocks, nblocks);
  if (threadIdx.x != 0) return;
  A.S[(size_t)k * kScal + SC_T2] = r2;
  reliable_decide(A.S, A.ctl, k, A.tol, A.hist, A.hist_its, A.hmax);
}

// The FP64 residual goes back into slot k of r (and, at a restart or with all set, of
// rhat); partial sums of <rhat, r>.
template <int P>
__global__ void __launch_bounds__(kPendThreads) pend_insert_kernel(PendArgs A, int mask) {
  const int k = blockIdx.y;
  if (!pend_on(A.ctl, mask, k)) return;
  using RB = typename SpinorIO<P>::R;
  const bool shadow = mask == PEND_ALL || ((A.ctl[CTL_RESTART] >> k) & 1u);
  const int s = blockIdx.x * kPendThreads + threadIdx.x;
  double re = 0.0, im = 0.0;
  if (s < A.vh) {
    const int e = s * A.nb + k, n = A.vh * A.nb;
    cplx<double> v[12];
    cplx<RB> r[12], h[12];
    SpinorIO<P64>::load(static_cast<const char*>(A.r64) + A.stride * k, nullptr, A.vh, s, v);
    if (!shadow) SpinorIO<P>::load(A.rhat.data, A.rhat.norm, n, e, h);
#pragma unroll
    for (int q = 0; q < 12; ++q) r[q] = {(RB)v[q].re, (RB)v[q].im};
    if (shadow) SpinorIO<P>::store(A.rhat.data, A.rhat.norm, n, e, r);
    SpinorIO<P>::store_rounded(A.r.data, A.r.norm, n, e, r);
    if (mask != PEND_ALL) {  // the product of what is stored
      if (shadow) {
#pragma unroll
        for (int q = 0; q < 12; ++q) h[q] = r[q];
      }
#pragma unroll
      for (int q = 0; q < 12; ++q) {
        re += (double)h[q].re * r[q].re + (double)h[q].im * r[q].im;
        im += (double)h[q].re * r[q].im - (double)h[q].im * r[q].re;
      }
    }
  }
  if (mask == PEND_ALL) return;
  __shared__ double red[2][kPendThreads / 32];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    re += __shfl_down_sync(0xffffffffu, re, o);
    im += __shfl_down_sync(0xffffffffu, im, o);
  }
  if ((threadIdx.x & 31) == 0) {
    red[0][threadIdx.x >> 5] = re;
    red[1][threadIdx.x >> 5] = im;
  }
  __syncthreads();
  if (threadIdx.x < 2) {
    double t = 0.0;
    for (int w = 0; w < kPendThreads / 32; ++w) t += red[threadIdx.x][w];
    A.partial[((size_t)k * 2 + threadIdx.x) * gridDim.x + blockIdx.x] = t;
  }
}

// rho' = <rhat, r> of the re-inserted residual, beta and rho (or, at a restart, rho =
// ||r||^2 and beta = 0), and right-hand side blockIdx.x iterates again.
__global__ void __launch_bounds__(256) pend_resume_kernel(PendArgs A, int nblocks) {
  const int k = blockIdx.x;
  const bool on = pend_on(A.ctl, PEND_INSERT, k);
  __syncthreads();
  if (!on) return;
  const double re = pend_sum(A.partial + (size_t)k * 2 * nblocks, nblocks);
  const double im = pend_sum(A.partial + ((size_t)k * 2 + 1) * nblocks, nblocks);
  if (threadIdx.x != 0) return;
  reliable_rho(A.S, A.ctl, k, re, im);
  reliable_resume(A.ctl, k);
}

// Partial sums (592 blocks) of |b - (x + tk J x - kappa h)|^2 and |b|^2: the residual is
// not stored.
__global__ void __launch_bounds__(kRedThreads) residual_norms_kernel(int vh, Spinor b, Spinor x, Spinor h, double tk,
                                                                     double kappa, double* partial) {
  double acc[3] = {0.0, 0.0, 0.0};
  for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < vh; s += gridDim.x * blockDim.x) {
    cplx<double> bv[12], xv[12], hv[12];
    SpinorIO<P64>::load(b.data, nullptr, vh, s, bv);
    SpinorIO<P64>::load(x.data, nullptr, vh, s, xv);
    SpinorIO<P64>::load(h.data, nullptr, vh, s, hv);
#pragma unroll
    for (int c = 0; c < 12; ++c) {
      const cplx<double> j = c < 6 ? xv[c + 6] : cplx<double>{-xv[c - 6].re, -xv[c - 6].im};
      const double re = bv[c].re - (xv[c].re + tk * j.re - kappa * hv[c].re);
      const double im = bv[c].im - (xv[c].im + tk * j.im - kappa * hv[c].im);
      acc[0] += re * re + im * im;
      acc[1] += bv[c].re * bv[c].re + bv[c].im * bv[c].im;
    }
  }
  block_reduce_store<3>(acc, partial);
}

template <int RES>
cudaError_t pend_hop(const HopArgs& h, const PendArgs& A, int recon, int epi, int mask, cudaStream_t st) {
  const dim3 grd((A.vh + kPendThreads - 1) / kPendThreads, A.nb);
  if (RES) epi = EPI_STORE;
  if (recon == 18)
    epi == EPI_TWIST ? pend_hop_kernel<18, EPI_TWIST, RES><<<grd, kPendThreads, 0, st>>>(h, A, mask)
                     : pend_hop_kernel<18, EPI_STORE, RES><<<grd, kPendThreads, 0, st>>>(h, A, mask);
  else
    epi == EPI_TWIST ? pend_hop_kernel<12, EPI_TWIST, RES><<<grd, kPendThreads, 0, st>>>(h, A, mask)
                     : pend_hop_kernel<12, EPI_STORE, RES><<<grd, kPendThreads, 0, st>>>(h, A, mask);
  return cudaGetLastError();
}

template <int P>
cudaError_t pend_field(const PendArgs& A, bool insert, int mask, cudaStream_t st) {
  const dim3 grd((A.vh + kPendThreads - 1) / kPendThreads, A.nb);
  if (insert)
    pend_insert_kernel<P><<<grd, kPendThreads, 0, st>>>(A, mask);
  else
    pend_accum_kernel<P><<<grd, kPendThreads, 0, st>>>(A);
  return cudaGetLastError();
}

cudaError_t pend_field(const PendArgs& A, int prec, bool insert, int mask, cudaStream_t st) {
  return prec == P32 ? pend_field<P32>(A, insert, mask, st)
         : prec == P16 ? pend_field<P16>(A, insert, mask, st)
         : prec == PB16 ? pend_field<PB16>(A, insert, mask, st) : pend_field<P64>(A, insert, mask, st);
}

// r64 = b - A x of the right-hand sides in `mask`, with the partial norms.
int pend_residual(qq_ctx* c, const PendArgs& A, const double kappa[2], int mask) {
  HopArgs h1, h2;
  int epi = EPI_STORE;
  hop_pair_args(c, P64, 0, kappa, &h1, &h2, &epi);
  count_launch(2);
  QQ_CK(pend_hop<0>(h1, A, c->recon64, epi, mask, c->st));
  QQ_CK(pend_hop<1>(h2, A, c->recon64, EPI_STORE, mask, c->st));
  return QQ_OK;
}

int pend_blocks(const PendArgs& A) { return (A.vh + kPendThreads - 1) / kPendThreads; }

}  // namespace

size_t pend_partials(int vh, int nb) { return (size_t)2 * nb * ((vh + kPendThreads - 1) / kPendThreads); }

int residual_norms(qq_ctx* c, Spinor b, Spinor x, Spinor h, double tk, double kappa, double* out) {
  double* part = c->partial.as<double>();
  count_launch();
  residual_norms_kernel<<<kRedBlocks, kRedThreads, 0, c->st>>>(c->g.vh, b, x, h, tk, kappa, part);
  QQ_CK(cudaGetLastError());
  QQ_CK(launch_finalize(part, kRedBlocks, 3, 2, out, 0, c->st));
  return QQ_OK;
}

int pend_start(qq_ctx* c, const PendArgs& A, int prec, const double kappa[2]) {
  QQ_TRY(pend_residual(c, A, kappa, PEND_ALL));
  count_launch(2);
  pend_init_kernel<<<A.nb, 256, 0, c->st>>>(A, pend_blocks(A));
  QQ_CK(cudaGetLastError());
  QQ_CK(pend_field(A, prec, true, PEND_ALL, c->st));
  return QQ_OK;
}

int pend_update(qq_ctx* c, const PendArgs& A, int prec, const double kappa[2]) {
  count_launch(4);
  QQ_CK(pend_field(A, prec, false, PEND_PENDING, c->st));
  QQ_TRY(pend_residual(c, A, kappa, PEND_PENDING));
  pend_decide_kernel<<<A.nb, 256, 0, c->st>>>(A, pend_blocks(A));
  QQ_CK(cudaGetLastError());
  QQ_CK(pend_field(A, prec, true, PEND_INSERT, c->st));
  pend_resume_kernel<<<A.nb, 256, 0, c->st>>>(A, pend_blocks(A));
  QQ_CK(cudaGetLastError());
  return QQ_OK;
}

}  // namespace qq

// Wilson loop operators of one noise with the perturbative subtraction levels of the
// Wilson driver (qq_average): average, Q/disconloops.f90:5343-5733, with loopops
// (:7769-7910) and spacesum (:9012-9124).
//
// Level 1 uses the solution x; level k >= 2 subtracts sub_k = sum_{n=0}^{k+1} kappa^n H^n b,
// the hopping expansion of the propagator applied to the noise b (H = Hsingle on each
// half).  For y = x - sub_k, a thread per site and direction evaluates loopops in closed
// form:
//   J_mu = conj( y(x+mu)^+ (1 - gamma_mu) U_mu(x)^+ b(x) - y(x)^+ (1 + gamma_mu) U_mu(x) b(x+mu) )
//   J_5 = conj(y^+ b) (+ 12 on levels k >= 2),  J_{5+mu} = conj(y^+ gamma_mu b),
// neighbours across the lattice edge times bc(mu), the complex noise kept whole.  Sums
// over (time slice, momentum) run in a fixed order: every operator at imom = 1, and the
// caller's momentum factors momfac(isite, ieo, ibl, imom-1, k) on operators 1..5 in
// spacesum's slots.  Operators 1..4 are then multiplied by kappa.
// The test suite checks this against the CPU restatement of the reference's loops,
// which is itself checked against an independent numpy statement.
//
// Everything runs on fields in the GPU layout: the noise and the solution are converted
// once, y is updated in place by each power of H, and nothing waits for the host between
// levels.  The momentum factors are the caller's host array; they are uploaded on the
// second stream while the levels run.  Six levels and five momenta at 16^3x32: 1.6 ms,
// where the expansion through reference-layout Hsingle calls took 6.0 ms.
#include <cmath>
#include <cstring>
#include <vector>

#include "qq_ctx.h"

namespace qq {
namespace {

constexpr int kAvVals = 18;     // 9 complex operators per site
constexpr int kAvMom = 7;       // of them in the momentum sums: values 1, 3, 5, 6..9
constexpr int kAvThreads = 128;

using C2 = cplx<double>;

// (1 + S gamma_MU) v as its two independent colour vectors (the factor 2 of MU = 3 left
// out); the product of two such half spinors is a^+ (1 + S gamma_MU) b, for MU = 3 half
// of it.
template <int MU, int S>
__device__ inline void half_spinor(const C2* v, C2* h) {
  constexpr double s = (double)S;
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    if (MU == 0) {
      h[c] = cadd(v[c], cscale(s, v[9 + c]));
      h[3 + c] = cadd(v[3 + c], cscale(s, v[6 + c]));
    } else if (MU == 1) {
      h[c] = csub(v[c], cscale(s, ctimesi(v[9 + c])));
      h[3 + c] = cadd(v[3 + c], cscale(s, ctimesi(v[6 + c])));
    } else if (MU == 2) {
      h[c] = cadd(v[c], cscale(s, v[6 + c]));
      h[3 + c] = csub(v[3 + c], cscale(s, v[9 + c]));
    } else {
      h[c] = S < 0 ? v[6 + c] : v[c];
      h[3 + c] = S < 0 ? v[9 + c] : v[3 + c];
    }
  }
}

template <int N>
__device__ inline C2 vdot(const C2* a, const C2* b) {  // a^+ b
  C2 s{0.0, 0.0};
#pragma unroll
  for (int c = 0; c < N; ++c) s = cadd(s, cmulconj(a[c], b[c]));
  return s;
}

// y^+ gamma_MU b, the gammas of Q/diracops.f90:61-71
template <int MU>
__device__ inline C2 gamma_dot(const C2* y, const C2* b) {
  if (MU == 0) return cadd(cadd(vdot<3>(y, b + 9), vdot<3>(y + 3, b + 6)), cadd(vdot<3>(y + 6, b + 3), vdot<3>(y + 9, b)));
  if (MU == 1)  // rows (-i, i, -i, i) of the reversed spins
    return ctimesi(cadd(csub(vdot<3>(y + 3, b + 6), vdot<3>(y, b + 9)), csub(vdot<3>(y + 9, b), vdot<3>(y + 6, b + 3))));
  if (MU == 2) return cadd(csub(vdot<3>(y, b + 6), vdot<3>(y + 3, b + 9)), csub(vdot<3>(y + 6, b), vdot<3>(y + 9, b + 3)));
  return csub(vdot<6>(y, b), vdot<6>(y + 6, b + 6));
}

struct LoopArgs {
  Geom g;
  Spinor y[2], b[2];  // per parity
  const void* gauge;
  int ksub;
  double* mom;      // [kAvMom][2 vh] per-site values of the momentum sums, or null
  double* partial;  // [nt][kAvVals][2 chunks]
};

// The site's values of direction MU: out[0..1] operator MU + 1, out[2..3] operator
// 6 + MU, out[4..5] (MU = 0) operator 5.
template <int MU, int RECON>
__device__ inline void loop_dir(const LoopArgs& A, int p, int s, double* out) {
  int x[4];
  site_coords(A.g, p, s, x);
  double f = MU == 3 ? 2.0 : 1.0;
  x[MU] += 1;
  if (x[MU] == A.g.n[MU]) {
    x[MU] = 0;
    f *= A.g.bcd[MU];
  }
  const int sn = site_index(A.g, x);
  C2 y[12], b[12], v[12], h[6], w[6], hy[6];
  Su3<double> u;
  LinkIO<P64, RECON>::load(A.gauge, A.g.vh, p, MU, s, u);
  SpinorIO<P64>::load(A.y[p].data, nullptr, A.g.vh, s, y);
  SpinorIO<P64>::load(A.b[p].data, nullptr, A.g.vh, s, b);
  const C2 gd = gamma_dot<MU>(y, b);
  out[2] = gd.re;
  out[3] = -gd.im;
  if (MU == 0) {
    const C2 s5 = vdot<12>(y, b);
    out[4] = s5.re + (A.ksub ? 12.0 : 0.0);
    out[5] = -s5.im;
  }
  // y(x+mu)^+ (1 - gamma) U^+ b(x)
  half_spinor<MU, -1>(b, h);
  matvec_dag(u, h, w);
  matvec_dag(u, h + 3, w + 3);
  SpinorIO<P64>::load(A.y[1 - p].data, nullptr, A.g.vh, sn, v);
  half_spinor<MU, -1>(v, hy);
  const C2 a0 = vdot<6>(hy, w);
  // y(x)^+ (1 + gamma) U b(x+mu)
  SpinorIO<P64>::load(A.b[1 - p].data, nullptr, A.g.vh, sn, v);
  half_spinor<MU, +1>(v, h);
  matvec(u, h, w);
  matvec(u, h + 3, w + 3);
  half_spinor<MU, +1>(y, hy);
  const C2 b0 = vdot<6>(hy, w);
  out[0] = f * (a0.re - b0.re);
  out[1] = -f * (a0.im - b0.im);
}

// Grid (32-site chunks of a slice's parity, nt, parity); warp mu of a block takes direction
// mu of its 32 sites (a slice's parity has a multiple of 32), so a site's spinors are read
// from HBM once and by the other directions from L1, and the sums need no shared memory.
template <int RECON>
__global__ void __launch_bounds__(kAvThreads) loopops_kernel(LoopArgs A) {
  const int vs = A.g.vh / A.g.n[3], t = blockIdx.y, p = blockIdx.z, mu = threadIdx.y;
  const int s = t * vs + blockIdx.x * 32 + threadIdx.x;
  double out[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
  switch (mu) {
    case 0: loop_dir<0, RECON>(A, p, s, out); break;
    case 1: loop_dir<1, RECON>(A, p, s, out); break;
    case 2: loop_dir<2, RECON>(A, p, s, out); break;
    default: loop_dir<3, RECON>(A, p, s, out); break;
  }
  if (A.mom) {
    const size_t V = 2 * (size_t)A.g.vh, e = (size_t)p * A.g.vh + s;
    if (mu < 3) {
      A.mom[mu * V + e] = out[1];
    } else {
      A.mom[3 * V + e] = out[0];
      A.mom[4 * V + e] = out[1];
    }
    if (mu == 0) {
      A.mom[5 * V + e] = out[4];
      A.mom[6 * V + e] = out[5];
    }
  }
  const int chunks = 2 * gridDim.x, chunk = p * gridDim.x + blockIdx.x;
#pragma unroll
  for (int k = 0; k < 6; ++k) {
    double v = out[k];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    const int row = k < 2 ? 2 * mu + k : k < 4 ? 10 + 2 * mu + k - 2 : 8 + k - 4;
    if (threadIdx.x == 0 && (k < 4 || mu == 0)) A.partial[((size_t)t * kAvVals + row) * chunks + chunk] = v;
  }
}

// spacesum's momentum slots (:9057-9085) for operators 1..5, imom >= 2: output (op, re/im)
// takes stored value src of the site times momfac component fac (1-based).  Grid (chunks of a slice, nt, level * (nmom - 1) + imom - 2):
// partial[((level * (nmom - 1) + imom - 2) * nt + t) * 10 + slot][chunk].
__global__ void __launch_bounds__(kAvThreads) momentum_kernel(Geom g, const double* mom, const double* momfac, int nmom,
                                                              double* partial) {
  const int nt = g.n[3], vs = g.vh / nt, t = blockIdx.y, im = blockIdx.z % (nmom - 1), lev = blockIdx.z / (nmom - 1);
  const size_t V = 2 * (size_t)g.vh, nvh = (size_t)g.vh / 16;  // nvh: the reference's nvhalf
  const size_t kstride = (size_t)(nmom - 1) * 32 * nvh;
  const double* val = mom + (size_t)lev * kAvMom * V;
  double acc[10];
#pragma unroll
  for (int k = 0; k < 10; ++k) acc[k] = 0.0;
  for (int i = blockIdx.x * kAvThreads + threadIdx.x; i < 2 * vs; i += gridDim.x * kAvThreads) {
    const int p = i >= vs, s = t * vs + (p ? i - vs : i);
    int x[4], isite, ieo, ibleo;
    site_coords(g, p, s, x);
    ref_site(g, x, &isite, &ieo, &ibleo);
    const int ibl = (x[0] & 1) + 2 * (x[1] & 1) + 4 * (x[2] & 1) + 8 * (x[3] & 1);
    const double* mf = momfac + (((size_t)im * 16 + ibl) * 2 + (ieo - 1)) * nvh + (isite - 1);
    double f[5], v[kAvMom];
#pragma unroll
    for (int k = 0; k < 5; ++k) f[k] = __ldg(mf + k * kstride);
#pragma unroll
    for (int k = 0; k < kAvMom; ++k) v[k] = __ldg(val + k * V + (size_t)p * g.vh + s);
    constexpr int src[10] = {0, 0, 1, 1, 2, 2, 3, 4, 5, 6}, fac[10] = {3, 2, 1, 3, 2, 1, 4, 4, 5, 5};
#pragma unroll
    for (int o = 0; o < 10; ++o) acc[o] += v[src[o]] * f[fac[o] - 1];
  }
  __shared__ double red[10][kAvThreads / 32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
  for (int k = 0; k < 10; ++k) {
    double v = acc[k];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if (lane == 0) red[k][wid] = v;
  }
  __syncthreads();
  if (threadIdx.x < 10) {
    double v = 0.0;
    for (int w = 0; w < kAvThreads / 32; ++w) v += red[threadIdx.x][w];
    partial[(((size_t)blockIdx.z * nt + t) * 10 + threadIdx.x) * gridDim.x + blockIdx.x] = v;
  }
}

// out[i] = sum_b partial[i * nb + b] in a fixed order, a warp per output
__global__ void __launch_bounds__(kAvThreads) loop_fold_kernel(const double* partial, int n, int nb, double* out) {
  const int i = (blockIdx.x * kAvThreads + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (i >= n) return;
  double s = 0.0;
  for (int b = lane; b < nb; b += 32) s += partial[(size_t)i * nb + b];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
  if (lane == 0) out[i] = s;
}

int loop_chunks(const Geom& g) { return g.vh / g.n[3] / 32; }

int loop_fold(qq_ctx* c, const double* partial, int n, int nb, double* out) {
  count_launch();
  loop_fold_kernel<<<(n * 32 + kAvThreads - 1) / kAvThreads, kAvThreads, 0, c->st>>>(partial, n, nb, out);
  QQ_CK(cudaGetLastError());
  return QQ_OK;
}

// Operators of y and b (per parity): slice sums out[t * kAvVals + k], and the values of
// the momentum sums when mom is given.  partial: nt * kAvVals * 2 chunks doubles.
int loopops(qq_ctx* c, const Spinor* y, const Spinor* b, int ksub, double* mom, double* partial, double* out) {
  LoopArgs A;
  A.g = c->g;
  for (int p = 0; p < 2; ++p) {
    A.y[p] = y[p];
    A.b[p] = b[p];
  }
  A.gauge = c->gauge64.p;
  A.ksub = ksub;
  A.mom = mom;
  A.partial = partial;
  const int nt = c->g.n[3];
  const dim3 grid(loop_chunks(c->g), nt, 2);
  count_launch();
  if (c->recon64 == 18)
    loopops_kernel<18><<<grid, dim3(32, 4), 0, c->st>>>(A);
  else
    loopops_kernel<12><<<grid, dim3(32, 4), 0, c->st>>>(A);
  QQ_CK(cudaGetLastError());
  return loop_fold(c, partial, nt * kAvVals, 2 * (int)grid.x, out);
}

enum WsId : int { WS_AV_MOM = 40, WS_AV_FAC, WS_AV_PART, WS_AV_SUMS };

}  // namespace

// Loop operators of y (solution side) and b (noise), even and odd halves, at zero
// momentum, summed per time slice, without the kappa factors: loopops with ksub, then
// spacesum at imom = 1.  J_host[(iop * nt + t) * 2 + ri], iop < 9.
int loop_slices(qq_ctx* c, const Spinor y[2], const Spinor b[2], int ksub, double* J_host) {
  const int nt = c->g.n[3];
  double *part = nullptr, *sums = nullptr;
  QQ_CK(ws_get(c, WS_AV_PART, sizeof(double) * nt * kAvVals * 2 * loop_chunks(c->g), reinterpret_cast<void**>(&part)));
  QQ_CK(ws_get(c, WS_AV_SUMS, sizeof(double) * nt * kAvVals, reinterpret_cast<void**>(&sums)));
  QQ_TRY(loopops(c, y, b, ksub, nullptr, part, sums));
  std::vector<double> h((size_t)nt * kAvVals);
  QQ_CK(cudaMemcpyAsync(h.data(), sums, sizeof(double) * h.size(), cudaMemcpyDeviceToHost, c->st));
  QQ_CK(cudaStreamSynchronize(c->st));
  for (int t = 0; t < nt; ++t)
    for (int k = 0; k < kAvVals; ++k) J_host[((size_t)(k / 2) * nt + t) * 2 + k % 2] = h[(size_t)t * kAvVals + k];
  return QQ_OK;
}

}  // namespace qq

using namespace qq;

extern "C" int qq_average(qq_ctx* c, const double* be, const double* bo, const double* xe, const double* xo,
                          double kappa, int nsub, int nmom, int nop, const double* momfac, double* Jtime) {
  if (!c) return set_error(QQ_BAD_ARG, "null context");
  if (!be || !bo || !xe || !xo || !Jtime) return set_error(QQ_BAD_ARG, "null argument");
  if (!c->have_gauge) return set_error(QQ_BAD_ARG, "no gauge field uploaded");
  if (nsub < 1 || nsub > 6) return set_error(QQ_BAD_ARG, "nsub must be 1..6");
  if (nmom < 1 || nmom > 5) return set_error(QQ_BAD_ARG, "nmom must be 1..5");
  if (nop < 9) return set_error(QQ_BAD_ARG, "nop must be at least 9");
  if (nmom > 1 && !momfac) return set_error(QQ_BAD_ARG, "momfac is needed for nmom > 1");
  QQ_CK(cudaSetDevice(c->device));
  const size_t nv = c->ref_doubles(), V = 2 * (size_t)c->g.vh;
  const int nt = c->g.n[3], vs = c->g.vh / nt;
  Tmp b0(c, P64), b1(c, P64), y0(c, P64), y1(c, P64), p0(c, P64), p1(c, P64), q0(c, P64), q1(c, P64);
  QQ_TRY(have({&b0, &b1, &y0, &y1, &p0, &p1, &q0, &q1}));
  const Spinor b[2] = {b0.sp(), b1.sp()}, y[2] = {y0.sp(), y1.sp()};
  const Spinor scratch[2][2] = {{p0.sp(), p1.sp()}, {q0.sp(), q1.sp()}};
  const double* src[4] = {be, bo, xe, xo};
  for (int i = 0; i < 4; ++i) {
    const double* d = nullptr;
    QQ_TRY(stage_in(c, i, src[i], nv, &d));
    QQ_TRY(ref_to_field(c, d, i & 1, i < 2 ? b[i] : y[i - 2]));
  }
  // scratch: values of the momentum sums per level, the factors, partial and slice sums
  const int nm = nmom - 1, chunks = loop_chunks(c->g), mchunks = (2 * vs + 4 * kAvThreads - 1) / (4 * kAvThreads);
  const size_t nmf = (size_t)5 * nm * 32 * (c->g.vh / 16);
  const size_t nsum0 = (size_t)nt * kAvVals, nsumm = (size_t)nsub * nm * nt * 10;
  double *mom = nullptr, *fac = nullptr, *part = nullptr, *sums = nullptr;
  if (nm) {
    QQ_CK(ws_get(c, WS_AV_MOM, sizeof(double) * kAvMom * V * nsub, reinterpret_cast<void**>(&mom)));
    QQ_CK(ws_get(c, WS_AV_FAC, sizeof(double) * nmf, reinterpret_cast<void**>(&fac)));
  }
  QQ_CK(ws_get(c, WS_AV_PART, sizeof(double) * std::max<size_t>(nsum0 * 2 * chunks, nsumm * mchunks),
               reinterpret_cast<void**>(&part)));
  QQ_CK(ws_get(c, WS_AV_SUMS, sizeof(double) * (nsum0 * nsub + nsumm), reinterpret_cast<void**>(&sums)));
  // power n of H on b, alternating between the scratch pairs; y -= kappa^n H^n b
  auto subtract = [&](int n) -> int {
    const Spinor* in = n == 1 ? b : scratch[n % 2];
    const Spinor* out = scratch[(n + 1) % 2];
    for (int p = 0; p < 2; ++p) {
      QQ_TRY(op_hsingle(c, out[p], in[1 - p], 0, p));
      QQ_TRY(lin(c, y[p], cimm(1.0), y[p], cimm(-std::pow(kappa, n)), out[p]));
    }
    return QQ_OK;
  };
  for (int isub = 1; isub <= nsub; ++isub) {
    if (isub == 2) {  // O(kappa^0) .. O(kappa^3), :5398-5489
      for (int p = 0; p < 2; ++p) QQ_TRY(lin(c, y[p], cimm(1.0), y[p], cimm(-1.0), b[p]));
      for (int n = 1; n <= 3; ++n) QQ_TRY(subtract(n));
    } else if (isub > 2) {  // O(kappa^(isub+1)), :5490-5614
      QQ_TRY(subtract(isub + 1));
    }
    QQ_TRY(loopops(c, y, b, isub > 1, mom ? mom + (size_t)(isub - 1) * kAvMom * V : nullptr, part,
                   sums + (size_t)(isub - 1) * nsum0));
  }
  if (nm) {
    if (!c->aux_st) QQ_CK(cudaStreamCreateWithFlags(&c->aux_st, cudaStreamNonBlocking));
    QQ_CK(cudaMemcpyAsync(fac, momfac, sizeof(double) * nmf, cudaMemcpyDefault, c->aux_st));
    QQ_CK(cudaEventRecord(c->ev0, c->aux_st));
    QQ_CK(cudaStreamWaitEvent(c->st, c->ev0, 0));
    count_launch();
    momentum_kernel<<<dim3(mchunks, nt, nsub * nm), kAvThreads, 0, c->st>>>(c->g, mom, fac, nmom, part);
    QQ_CK(cudaGetLastError());
    QQ_TRY(loop_fold(c, part, (int)nsumm, mchunks, sums + nsum0 * nsub));
  }
  std::vector<double> h(nsum0 * nsub + nsumm), out((size_t)2 * nt * nsub * nmom * nop, 0.0);
  QQ_CK(cudaMemcpyAsync(h.data(), sums, sizeof(double) * h.size(), cudaMemcpyDeviceToHost, c->st));
  QQ_CK(cudaStreamSynchronize(c->st));
  for (int iop = 0; iop < 9; ++iop)
    for (int im = 0; im < nmom; ++im) {
      if (im > 0 && iop >= 5) break;
      for (int lev = 0; lev < nsub; ++lev)
        for (int t = 0; t < nt; ++t)
          for (int ri = 0; ri < 2; ++ri) {
            const double v = im == 0 ? h[(size_t)lev * nsum0 + (size_t)t * kAvVals + 2 * iop + ri]
                                     : h[nsum0 * nsub + (((size_t)lev * nm + im - 1) * nt + t) * 10 + 2 * iop + ri];
            // operators 1..4 times kappa (:5728-5731)
            out[((((size_t)iop * nmom + im) * nsub + lev) * nt + t) * 2 + ri] = iop < 4 ? kappa * v : v;
          }
    }
  QQ_CK(cudaMemcpy(Jtime, out.data(), sizeof(double) * out.size(), cudaMemcpyDefault));
  return QQ_OK;
}

// momfacs, Q/disconloops.f90:8925-8984 (host only): the momentum factors qq_average
// takes, momfac(nvhalf, 2, 16, 4, 5), nvhalf = nx ny nz nt / 32.  The reference's twoPi
// is a default-kind literal, so it carries the single-precision value.
extern "C" int qq_momfacs(const int dims[4], const int io[3], double* momfac) {
  if (!dims || !io || !momfac) return set_error(QQ_BAD_ARG, "null argument");
  Geom g{};
  for (int d = 0; d < 4; ++d) {
    if (dims[d] < 4 || dims[d] % 4 != 0) return set_error(QQ_BAD_ARG, "lattice extents must be multiples of 4");
    g.n[d] = dims[d];
    g.bc[d] = 1;
  }
  geom_finish(g);
  const int nx = dims[0], ny = dims[1], nz = dims[2], nt = dims[3];
  const size_t nv = (size_t)nx * ny * nz * nt / 32;
  const double twoPi = (double)6.283185307179586f;
  auto M = [&](int isite, int ieo, int ibl, int im, int k) -> double& {
    return momfac[((((size_t)(k - 1) * 4 + (im - 1)) * 16 + (ibl - 1)) * 2 + (ieo - 1)) * nv + (isite - 1)];
  };
  for (int it = 1; it <= nt; ++it)
    for (int iz = 1; iz <= nz; ++iz) {
      const double dz = twoPi * (double)(iz - io[2]) / (double)nz;
      for (int iy = 1; iy <= ny; ++iy) {
        const double dy = twoPi * (double)(iy - io[1]) / (double)ny;
        for (int ix = 1; ix <= nx; ++ix) {
          const double dx = twoPi * (double)(ix - io[0]) / (double)nx;
          const int x[4] = {ix - 1, iy - 1, iz - 1, it - 1};
          int isite, ieo, ibleo;
          ref_site(g, x, &isite, &ieo, &ibleo);
          const int ibl = 1 + (x[0] & 1) + 2 * (x[1] & 1) + 4 * (x[2] & 1) + 8 * (x[3] & 1);
          const double cx = std::cos(dx), cy = std::cos(dy), cz = std::cos(dz);
          const double sx = std::sin(dx), sy = std::sin(dy), sz = std::sin(dz);
          const double v[4][4] = {{sx, sy, sz, (cx + cy + cz) / 3.0},
                                  {sx * (cy + cz) / 2.0, sy * (cx + cz) / 2.0, sz * (cx + cy) / 2.0,
                                   (cx * cy + cx * cz + cy * cz) / 3.0},
                                  {sx * cy * cz, sy * cx * cz, sz * cx * cy, cx * cy * cz},
                                  {std::sin(2.0 * dx), std::sin(2.0 * dy), std::sin(2.0 * dz),
                                   (std::cos(2.0 * dx) + std::cos(2.0 * dy) + std::cos(2.0 * dz)) / 3.0}};
          for (int im = 1; im <= 4; ++im) {
            for (int k = 1; k <= 4; ++k) M(isite, ieo, ibl, im, k) = v[im - 1][k - 1];
            M(isite, ieo, ibl, im, 5) = v[im - 1][3];
          }
        }
      }
    }
  return QQ_OK;
}

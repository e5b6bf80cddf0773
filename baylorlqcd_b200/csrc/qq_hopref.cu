// The FP64 hopping term on fields in the reference's layout, for single applications of
// the operator: the first hop reads the caller's array and the last one writes it, so the
// conversions to and from the GPU layout are neither launches nor passes of their own.
// A spin's row of the reference layout is 48 contiguous bytes, three 16-byte vectors, and
// neighbouring sites of a checkerboard block follow each other; the blocks' interleaving
// costs L1 requests, of which the FP64 hop has to spare.  Solvers, which apply the operator
// many times to one field, convert once instead.  Hdbletm through the GPU layout took 35 us
// at 8^4, 39.6 at 12x20x4x28 and 253 at 24^3x48; this way 21.8, 27.3 and 203.
#include "qq_ctx.h"

namespace qq {
namespace {

// Where a site's spinor lies: the first vector of spin 1, and the vectors between spins.
struct RefField {
  double2* p;
  RefDims d;
  __device__ size_t row(const Geom& g, const int* x) const {
    int isite, ieo, ibleo;
    ref_site(g, x, &isite, &ieo, &ibleo);
    return ref_gi(d, 1, isite, 1, ieo, ibleo) / 2;
  }
  // spins LO .. LO + N - 1
  template <int LO, int N>
  __device__ void load(size_t row, cplx<double>* v) const {
#pragma unroll
    for (int id = LO; id < LO + N; ++id)
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const double2 t = __ldg(p + row + (size_t)id * 3 * d.ntotal + c);
        v[3 * id + c] = {t.x, t.y};
      }
  }
  __device__ void store(size_t row, const cplx<double>* v) const {
#pragma unroll
    for (int id = 0; id < 4; ++id)
#pragma unroll
      for (int c = 0; c < 3; ++c)
        p[row + (size_t)id * 3 * d.ntotal + c] = make_double2(v[3 * id + c].re, v[3 * id + c].im);
  }
};

struct RefHop {
  RefField in, out, aux;
};

// IN / OUT: the input / the output (and EPI_DBLE's operand) is in the reference layout.
// Thread layout of hop_kernel for one right-hand side: TPS direction groups per site.  A
// thread per site has its registers capped for three blocks per SM (uncapped, 226
// registers and two blocks: 39.1 us against 40.5 for Hdbletm on 24,576 sites of a parity,
// 55.4 against 43.0 on 40,960, 234 against 199 on 331,776).
template <int RECON, int TPS, int EPI, bool IN, bool OUT>
__global__ void __launch_bounds__(128, TPS == 1 ? 3 : 1) hop_ref_kernel(HopArgs a, RefHop f) {
  const int tx = threadIdx.x, ty = threadIdx.y;
  const int s = blockIdx.x * blockDim.x + tx;
  const bool active = s < a.g.vh;
  cplx<double> acc[12];
#pragma unroll
  for (int c = 0; c < 12; ++c) acc[c] = {0.0, 0.0};
  int x[4] = {0, 0, 0, 0};
  if (OUT && ty == 0) {  // zeros in the halo slots, as Hsingle's `gout = 0.0_KR` leaves them
    const int nb = f.out.d.ntotal - f.out.d.nvhalf, total = nb * 3 * 4 * 2 * 8;
    for (int t = s; t < total; t += gridDim.x * blockDim.x) {
      int r = t;
      const int c = r % 3; r /= 3;
      const int ib = r % nb; r /= nb;
      const int id = r % 4; r /= 4;
      f.out.p[ref_gi(f.out.d, 2 * c + 1, f.out.d.nvhalf + ib + 1, id + 1, r % 2 + 1, r / 2 + 1) / 2] =
          make_double2(0.0, 0.0);
    }
  }
  if (active) {
    site_coords(a.g, a.pout, s, x);
    auto load = [&](const int* y, int sy, int half, cplx<double>* psi) {
      if (IN) {
        const size_t row = f.in.row(a.g, y);
        if (half == 0)
          f.in.load<0, 2>(row, psi);
        else if (half == 1)
          f.in.load<2, 2>(row, psi);
        else
          f.in.load<0, 4>(row, psi);
      } else if (half == 0) {
        load_half<P64, 0>(a.in[0], a.g.vh, sy, psi);
      } else if (half == 1) {
        load_half<P64, 1>(a.in[0], a.g.vh, sy, psi);
      } else {
        SpinorIO<P64>::load(a.in[0], nullptr, a.g.vh, sy, psi);
      }
    };
    if (TPS == 1 || ty == 0) {
      hop_from<P64, P64, RECON, 0, true>(a, s, x, acc, load);
      hop_from<P64, P64, RECON, 0, false>(a, s, x, acc, load);
    }
    if (TPS == 1 || ty == 1 % TPS) {
      hop_from<P64, P64, RECON, 1, true>(a, s, x, acc, load);
      hop_from<P64, P64, RECON, 1, false>(a, s, x, acc, load);
    }
    if (TPS == 1 || ty == 2 % TPS) {
      hop_from<P64, P64, RECON, 2, true>(a, s, x, acc, load);
      hop_from<P64, P64, RECON, 2, false>(a, s, x, acc, load);
    }
    if (TPS == 1 || ty == 3 % TPS) {
      hop_from<P64, P64, RECON, 3, true>(a, s, x, acc, load);
      hop_from<P64, P64, RECON, 3, false>(a, s, x, acc, load);
    }
  }
  if (TPS > 1) {
    __shared__ cplx<double> red[TPS > 1 ? 128 : 1][12];
    const int slot = ty * blockDim.x + tx;
    if (ty > 0) {
#pragma unroll
      for (int c = 0; c < 12; ++c) red[slot][c] = acc[c];
    }
    __syncthreads();
    if (ty > 0) return;
#pragma unroll
    for (int g = 1; g < TPS; ++g)
#pragma unroll
      for (int c = 0; c < 12; ++c) acc[c] = cadd(acc[c], red[g * blockDim.x + tx][c]);
  }
  if (!active) return;
  if (!OUT) return hop_finish<P64, EPI>(a, s, 0, acc);
  cplx<double> o[12], gg[12];
  const size_t row = f.out.row(a.g, x);
  if (EPI == EPI_DBLE) f.aux.load<0, 4>(row, gg);  // the same dimensions, hence the same row
  hop_combine<EPI>(a, acc, gg, o);
  f.out.store(row, o);
}

template <int RECON, int EPI, bool IN, bool OUT>
cudaError_t hop_ref_tps(const HopArgs& a, const RefHop& f, int tps, cudaStream_t st) {
  const dim3 blk(128 / tps, tps), grd((a.g.vh + blk.x - 1) / blk.x);
  switch (tps) {
    case 1: hop_ref_kernel<RECON, 1, EPI, IN, OUT><<<grd, blk, 0, st>>>(a, f); break;
    case 2: hop_ref_kernel<RECON, 2, EPI, IN, OUT><<<grd, blk, 0, st>>>(a, f); break;
    case 4: hop_ref_kernel<RECON, 4, EPI, IN, OUT><<<grd, blk, 0, st>>>(a, f); break;
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

template <int EPI, bool IN, bool OUT>
cudaError_t hop_ref(const HopArgs& a, const RefHop& f, int recon, int tps, cudaStream_t st) {
  return recon == 18 ? hop_ref_tps<18, EPI, IN, OUT>(a, f, tps, st) : hop_ref_tps<12, EPI, IN, OUT>(a, f, tps, st);
}

// Threads per site.  A site's hops in sequence are a chain of loads, so groups of
// directions side by side win as long as all the blocks run at once: 2 blocks per SM hold
// 148 * 2 * 128 threads, 9472 sites in four groups and 18,944 in two.  Hdbletm with a cold
// L2, four / two / one, in us: 2048 sites of a parity 28 / 30 / 36, 8192 31 / 31 / 37,
// 13,440 40 / 33 / 35, 18,432 42 / 34 / 38, 20,480 48 / 43 / 40, 36,864 61 / 47 / 40,
// 98,304 128 / 104 / 78.  Two groups start at 4096, where the fields that a caller has
// just touched are in L2 and they are the faster ones (27 against 28; 6144: 28 / 30).
int ref_tps(int vh) { return vh < 4096 ? 4 : vh <= 148 * 2 * 64 ? 2 : 1; }

bool aligned16(const void* p) { return reinterpret_cast<uintptr_t>(p) % 16 == 0; }

bool disjoint(const double* a, const double* b, size_t n) { return a + n <= b || b + n <= a; }

RefField ref_field(qq_ctx* c, const double* p) {
  return RefField{reinterpret_cast<double2*>(const_cast<double*>(p)), c->rd};
}

}  // namespace

bool hop_ref_usable(qq_ctx* c, const double* out, const double* in) {
  return aligned16(out) && aligned16(in) && disjoint(out, in, c->ref_doubles()) && !c->prof_hop && !c->forced_tps;
}

int op_hsingle_ref(qq_ctx* c, double* out, const double* in, int idag, int pout) {
  if (!c->have_gauge) return set_error(QQ_BAD_ARG, "no gauge field uploaded");
  const double none[2] = {1.0, 0.0};
  HopArgs a, b;
  int epi = EPI_STORE;
  hop_pair_args(c, P64, idag, none, &a, &b, &epi);
  a.pout = pout;
  const RefHop f{ref_field(c, in), ref_field(c, out), ref_field(c, nullptr)};
  count_launch();
  QQ_CK((hop_ref<EPI_STORE, true, true>(a, f, c->recon64, ref_tps(c->g.vh), c->st)));
  return QQ_OK;
}

int op_dbletm_ref(qq_ctx* c, double* out, const double* in, Spinor tmp, int idag, const double kappa[2]) {
  if (!c->have_gauge) return set_error(QQ_BAD_ARG, "no gauge field uploaded");
  HopArgs a, b;
  int epi = EPI_STORE;
  hop_pair_args(c, P64, idag, kappa, &a, &b, &epi);
  a.out[0] = tmp.data;
  b.in[0] = tmp.data;
  const RefHop f{ref_field(c, in), ref_field(c, out), ref_field(c, in)};
  const int tps = ref_tps(c->g.vh);
  count_launch(2);
  if (epi == EPI_TWIST)
    QQ_CK((hop_ref<EPI_TWIST, true, false>(a, f, c->recon64, tps, c->st)));
  else
    QQ_CK((hop_ref<EPI_STORE, true, false>(a, f, c->recon64, tps, c->st)));
  QQ_CK((hop_ref<EPI_DBLE, false, true>(b, f, c->recon64, tps, c->st)));
  return QQ_OK;
}

}  // namespace qq

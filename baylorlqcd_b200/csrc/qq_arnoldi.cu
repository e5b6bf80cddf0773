// Orthonormalisation of one Krylov vector against the basis.
//
// Classical Gram-Schmidt with one re-orthogonalisation needs h = V^H w, w' = w - V h,
// h2 = V^H w' and w'' = w' - V h2: four passes over the basis when every step is a kernel
// of its own, and all of them run at the memory's rate.  The two middle steps are one
// kernel here: three passes.  The middle one goes through the elements backwards, so the
// end of each pass is still in L2 when the next begins.
//
// The norm of w'' is taken from Pythagoras, ||w''||^2 = ||w'||^2 - ||h2||^2, as long as
// the second correction is small (||h2||^2 <= ||w'||^2 / 4: one bit of the sum at most is
// lost), so the last pass normalises as it writes; otherwise its last block divides by the
// norm summed from w'' itself.
//
// At 16^3x32 an iteration with 40 vectors spent 93 + 112 us on each of two products and
// two updates; the three passes take 93, 113 and 100 us.  At 8^4 eleven launches an
// iteration became seven.  An FP32 basis of 32 and more vectors spills some 500 bytes in the
// middle pass and gains all the same: a deflated batch of one source (m = 60, k = 20) at
// 16^3x32 50.0 -> 42.0 ms and at 24^3x48 187 -> 147, with m = 100, k = 40 55.3 -> 50.8 and
// 228 -> 200.
#include "qq_ctx.h"

namespace qq {
namespace {

constexpr int kOrthThreads = 128;
constexpr int kOrthWarps = kOrthThreads / 32;
constexpr int kOrthMaxVec = 127;
constexpr int kOrthMaxBlocks = 4 * 148;
static_assert(kOrthMaxBlocks * (2 * kOrthMaxVec + 1) <= kRedBlocks * 256, "partials exceed the context's buffer");

// Elements above which the first products of 32 or more vectors go to multidot_kernel:
// sixteen columns a lane leave 12 warps on an SM, too few for plain streaming (16^3x32, 40
// vectors: 111 us against 93); on lattices that fit the caches it is the faster one (8^4,
// 30 vectors: 6 us against 16).
constexpr size_t kOrthLarge = (size_t)1 << 19;

struct OrthArgs {
  const void* V;
  size_t stride, nel;  // 16-byte elements
  int nv;
  void* w;
  const double* h;     // ORTH_MID: V^H w.  ORTH_LAST: V^H w' and ||w'||^2
  double* hcol;        // column of H (may be null): V^H w, receives h + h2 and the norm
  double* part;
  unsigned* done;      // ORTH_LAST: blocks done, zero before and after
};

enum OrthStep : int {
  ORTH_FIRST = 0,  // V^H w
  ORTH_MID = 1,    // w' = w - V h, stored; V^H w' and ||w'||^2
  ORTH_LAST = 2,   // w'' = w' - V h2, normalised and stored
};

// ||h2||^2 in a fixed order, the same in every thread.
__device__ inline double orth_correction(const double* h2, int nv) {
  double s = 0.0;
  for (int v = threadIdx.x & 31; v < 2 * nv; v += 32) s += h2[v] * h2[v];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  return s;
}

// One pass.  A warp takes a tile of 32 / CG elements; lane (g, e) holds columns g, g + CG,
// ... of element e in registers, for the update and for the products, so a few shuffles
// are all that joins the lanes: no barriers, and the warps of an SM overlap each other's
// loads and sums.  (Tiles shared by a block's warps, in registers or in shared memory, met
// at two or three barriers each and ran at 2 to 4 TB/s; this runs at 5 to 5.7.)  w is
// column nv, with the coefficient -1.  A lane holds eight columns (up to 31 vectors) or
// sixteen, and the groups are as few as that allows: they cut the contiguous part of a
// column to 512 / CG bytes.  Products: per-block partials part[block * (2 nv + 1) + v].
template <int PB, int CG, int COLS, int STEP>
__global__ void __launch_bounds__(kOrthThreads, COLS == 8 ? 4 : 3) orth_kernel(OrthArgs a) {
  using IO = BasisIO<PB>;
  using T = typename IO::V;
  constexpr int C = IO::ncpx, EL = 32 / CG;
  __shared__ double2 hs[CG * COLS];
  __shared__ double2 sum[kOrthWarps][CG * COLS];
  __shared__ double nsum[kOrthWarps];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nv = a.nv, el = lane % EL, g = lane / EL;
  double scale = 1.0, norm = 0.0;
  bool direct = false;
  if (STEP != ORTH_FIRST) {
    for (int i = threadIdx.x; i < CG * COLS; i += kOrthThreads)
      hs[i] = i < nv ? make_double2(a.h[2 * i], a.h[2 * i + 1]) : make_double2(i == nv ? -1.0 : 0.0, 0.0);
    if (STEP == ORTH_LAST) {
      const double n2 = a.h[2 * nv], corr = orth_correction(a.h, nv);
      direct = !(corr <= 0.25 * n2);
      norm = sqrt(n2 - corr);
      if (!direct) scale = 1.0 / norm;
    }
    __syncthreads();
  }
  const int ntiles = (int)(a.nel / EL);  // a parity has a multiple of 128 sites
  const int first = blockIdx.x * kOrthWarps + warp, step = gridDim.x * kOrthWarps;
  const int mine = first < ntiles ? (ntiles - 1 - first) / step + 1 : 0;
  const T* const vb = static_cast<const T*>(a.V) + (size_t)g * a.stride + el;
  T* const wb = static_cast<T*>(a.w) + el;
  cplx<double> acc[COLS];
#pragma unroll
  for (int c = 0; c < COLS; ++c) acc[c] = {0.0, 0.0};
  double n2 = 0.0;
  for (int k = 0; k < mine; ++k) {
    const size_t e = (size_t)(first + (STEP == ORTH_MID ? mine - 1 - k : k) * step) * EL;
    T cur[COLS];
#pragma unroll
    for (int c = 0; c < COLS; ++c) {
      const int i = g + CG * c;
      cur[c] = T{};
      if (STEP == ORTH_FIRST ? i < nv : i <= nv) cur[c] = i == nv ? wb[e] : vb[(size_t)(CG * c) * a.stride + e];
    }
    cplx<double> x[C];
    if (STEP == ORTH_FIRST) {
      IO::ld(wb, e, x);
    } else {
#pragma unroll
      for (int q = 0; q < C; ++q) x[q] = {0.0, 0.0};
#pragma unroll
      for (int c = 0; c < COLS; ++c) {
        cplx<double> v[C];
        IO::ld(&cur[c], 0, v);
        const double2 h = hs[g + CG * c];
#pragma unroll
        for (int q = 0; q < C; ++q) {
          x[q].re -= h.x * v[q].re - h.y * v[q].im;
          x[q].im -= h.x * v[q].im + h.y * v[q].re;
        }
      }
#pragma unroll
      for (int o = EL; o < 32; o <<= 1)
#pragma unroll
        for (int q = 0; q < C; ++q) {
          x[q].re += __shfl_xor_sync(0xffffffffu, x[q].re, o);
          x[q].im += __shfl_xor_sync(0xffffffffu, x[q].im, o);
        }
      if (STEP == ORTH_MID && PB == P32)  // as stored
#pragma unroll
        for (int q = 0; q < C; ++q) x[q] = {(double)(float)x[q].re, (double)(float)x[q].im};
      if (g == 0) {
#pragma unroll
        for (int q = 0; q < C; ++q) {
          n2 += x[q].re * x[q].re + x[q].im * x[q].im;
          if (STEP == ORTH_LAST) x[q] = cscale(scale, x[q]);
        }
        IO::st(wb, e, x);
      }
    }
    if (STEP != ORTH_LAST) {
#pragma unroll
      for (int c = 0; c < COLS; ++c) {
        cplx<double> v[C];
        IO::ld(&cur[c], 0, v);
#pragma unroll
        for (int q = 0; q < C; ++q) {
          acc[c].re += v[q].re * x[q].re + v[q].im * x[q].im;
          acc[c].im += v[q].re * x[q].im - v[q].im * x[q].re;
        }
      }
    }
  }
  if (STEP != ORTH_FIRST) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) n2 += __shfl_xor_sync(0xffffffffu, n2, o);
    if (lane == 0) nsum[warp] = n2;
  }
  if (STEP != ORTH_LAST) {
#pragma unroll
    for (int c = 0; c < COLS; ++c) {
#pragma unroll
      for (int o = EL / 2; o > 0; o >>= 1) {
        acc[c].re += __shfl_xor_sync(0xffffffffu, acc[c].re, o);
        acc[c].im += __shfl_xor_sync(0xffffffffu, acc[c].im, o);
      }
      if (el == 0) sum[warp][g + CG * c] = make_double2(acc[c].re, acc[c].im);
    }
    __syncthreads();
    double* out = a.part + (size_t)blockIdx.x * (2 * nv + 1);
    for (int i = threadIdx.x; i < nv; i += kOrthThreads) {
      double2 s = make_double2(0.0, 0.0);
      for (int k = 0; k < kOrthWarps; ++k) {
        s.x += sum[k][i].x;
        s.y += sum[k][i].y;
      }
      out[2 * i] = s.x;
      out[2 * i + 1] = s.y;
    }
    if (STEP == ORTH_MID && threadIdx.x == 0) {
      double s = 0.0;
      for (int k = 0; k < kOrthWarps; ++k) s += nsum[k];
      out[2 * nv] = s;
    }
    return;
  }
  if (a.hcol && blockIdx.x == 0) {
    for (int v = threadIdx.x; v < 2 * nv; v += kOrthThreads) a.hcol[v] += a.h[v];
    if (threadIdx.x == 0) {
      a.hcol[2 * nv] = norm;
      a.hcol[2 * nv + 1] = 0.0;
    }
  }
  if (!direct) return;  // the same in every block
  __shared__ bool last;
  __syncthreads();
  if (threadIdx.x == 0) {
    double s = 0.0;
    for (int k = 0; k < kOrthWarps; ++k) s += nsum[k];
    a.part[blockIdx.x] = s;
    __threadfence();
    last = atomicAdd(a.done, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  double s = 0.0;
  for (int b = lane; b < gridDim.x; b += 32) s += __ldcg(a.part + b);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  norm = sqrt(s);
  for (size_t e = threadIdx.x; e < a.nel; e += kOrthThreads) {
    const T t = __ldcg(static_cast<const T*>(a.w) + e);
    cplx<double> x[C];
    IO::ld(&t, 0, x);
#pragma unroll
    for (int q = 0; q < C; ++q) x[q] = cscale(1.0 / norm, x[q]);
    IO::st(static_cast<T*>(a.w), e, x);
  }
  if (threadIdx.x == 0) {
    if (a.hcol) a.hcol[2 * nv] = norm;
    *a.done = 0u;
  }
}

template <int PB, int STEP>
int orth_pass(qq_ctx* c, const OrthArgs& a, int blocks) {
  count_launch();
  if (a.nv < 8)
    orth_kernel<PB, 1, 8, STEP><<<blocks, kOrthThreads, 0, c->st>>>(a);
  else if (a.nv < 16)
    orth_kernel<PB, 2, 8, STEP><<<blocks, kOrthThreads, 0, c->st>>>(a);
  else if (a.nv < 32)
    orth_kernel<PB, 4, 8, STEP><<<blocks, kOrthThreads, 0, c->st>>>(a);
  else if (a.nv < 64)
    orth_kernel<PB, 4, 16, STEP><<<blocks, kOrthThreads, 0, c->st>>>(a);
  else
    orth_kernel<PB, 8, 16, STEP><<<blocks, kOrthThreads, 0, c->st>>>(a);
  QQ_CK(cudaGetLastError());
  return QQ_OK;
}

template <int PB>
int orthonormalize(qq_ctx* c, const BasisArgs& V, int nv, void* w, double* hcol, double* h, double* h2,
                   unsigned* done) {
  OrthArgs a{V.base, V.stride, V.nel, nv, w, h, hcol, c->partial.as<double>(), done};
  // four blocks per SM (three at sixteen columns a lane); on small lattices two tiles a warp
  const size_t tiles = V.nel * (nv < 8 ? 1 : nv < 16 ? 2 : nv < 64 ? 4 : 8) / 32;
  const int blocks = (int)std::max<size_t>(1, std::min<size_t>((nv < 32 ? 4 : 3) * 148, tiles / (2 * kOrthWarps)));
  if (nv >= 32 && V.nel > kOrthLarge) {
    int ng = 0;
    QQ_CK(launch_multidot(PB, V, nv, w, a.part, &ng, c->st));
    QQ_CK(launch_finalize(a.part, kRedBlocks, ng * 16, 2 * nv, h, 0, c->st));
  } else {
    QQ_TRY((orth_pass<PB, ORTH_FIRST>(c, a, blocks)));
    QQ_CK(launch_finalize(a.part, blocks, 2 * nv + 1, 2 * nv, h, 0, c->st));
  }
  QQ_TRY((orth_pass<PB, ORTH_MID>(c, a, blocks)));
  QQ_CK(launch_finalize(a.part, blocks, 2 * nv + 1, 2 * nv + 1, h2, 0, c->st));
  a.h = h2;
  return orth_pass<PB, ORTH_LAST>(c, a, blocks);
}

}  // namespace

int op_orthonormalize(qq_ctx* c, int pb, const BasisArgs& V, int nv, void* w, double* hcol, double* ws) {
  if (nv < 1 || nv > kOrthMaxVec || V.nel % 32) return set_error(QQ_BAD_ARG, "basis too large or ragged");
  double *h = hcol ? hcol : ws, *h2 = ws + 2 * (kOrthMaxVec + 1);
  unsigned* done = reinterpret_cast<unsigned*>(ws + 4 * (kOrthMaxVec + 1));
  if (pb == P64) return orthonormalize<P64>(c, V, nv, w, hcol, h, h2, done);
  if (pb == P32) return orthonormalize<P32>(c, V, nv, w, hcol, h, h2, done);
  return set_error(QQ_BAD_ARG, "basis precision");
}

}  // namespace qq

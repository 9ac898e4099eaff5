// evolve.cu -- one Hamiltonian step of the class API in one launch:
//   psi <- B[ w(x) . F[psi] ]            (Potential / Interaction::Evolve)
//   fld <- (1 + F[ c(p) . B[phi] ]) / V  (Interaction::Initialize)
// for lattices that fit the shared memory of a CTA, one orbital per CTA.
//
// The reference's drivers step one configuration of a few orbitals at a time
// (src/hamiltonian/cuda/hamiltonian_evolve.cu), where a step made of pencil
// passes is a chain of seven (nine for Initialize) small launches, each with a
// trip of the orbitals through L2: the launches, 2-5 us each on the host, are
// the time.  Here the transforms along z, y and x run in place in shared
// memory (rows padded by one element), a thread per pencil, the x pass with
// the factor and the way back in one; the factors are applied as the pencil
// passes apply them.  7 FP32 orbitals of 24 x 12 x 16: 14 us a call against 37
// for the chain, Initialize on the same lattice 18 against 42.  The transforms'
// lengths are known at run time only, so each pass is a call of the function
// compiled for its length.
#include "common.cuh"
#include "fft.cuh"

namespace nrcps {

namespace {

enum EvolveOp { EV_NONE = 0, EV_COMPLEX = 1, EV_REAL = 2 };

// Pencil p of a pass starts at element (p / inner) * outer + p % inner of the
// padded array; its elements are `stride` apart.  Sites of an x pencil are p +
// j * plane.
struct EvolvePass {
  int pencils, inner, outer, stride, plane;
};

// DFT of every pencil; with an OP the transform, times the factor of each
// site, and the transform back
template <typename R, int N, int SIGN, int OP>
__device__ __noinline__ void evolve_pass(cplx<R>* sm, EvolvePass g, const double* __restrict__ table) {
  for (int p = threadIdx.x; p < g.pencils; p += blockDim.x) {
    cplx<R>* s = sm + (p / g.inner) * g.outer + p % g.inner;
    cplx<R> x[N];
#pragma unroll
    for (int j = 0; j < N; ++j) x[j] = s[j * g.stride];
    fft::Dft<N, SIGN, R>::run(x);
    if constexpr (OP == EV_COMPLEX) {
#pragma unroll
      for (int j = 0; j < N; ++j) {
        const double2 f = __ldg(reinterpret_cast<const double2*>(table) + p + j * g.plane);
        x[j] = cmul(cplx<R>{(R)f.x, (R)f.y}, x[j]);
      }
    } else if constexpr (OP == EV_REAL) {
#pragma unroll
      for (int j = 0; j < N; ++j) {
        const R k = (R)__ldg(table + p + j * g.plane);
        x[j] = cplx<R>{x[j].re * k, x[j].im * k};
      }
    }
    if constexpr (OP != EV_NONE) fft::Dft<N, -SIGN, R>::run(x);
#pragma unroll
    for (int j = 0; j < N; ++j) s[j * g.stride] = x[j];
  }
  __syncthreads();
}

template <typename R, int SIGN, int OP>
__device__ __forceinline__ void evolve_axis(int n, cplx<R>* sm, EvolvePass g, const double* table) {
  switch (n) {
    case 2: evolve_pass<R, 2, SIGN, OP>(sm, g, table); break;
    case 4: evolve_pass<R, 4, SIGN, OP>(sm, g, table); break;
    case 6: evolve_pass<R, 6, SIGN, OP>(sm, g, table); break;
    case 8: evolve_pass<R, 8, SIGN, OP>(sm, g, table); break;
    case 12: evolve_pass<R, 12, SIGN, OP>(sm, g, table); break;
    case 16: evolve_pass<R, 16, SIGN, OP>(sm, g, table); break;
    case 24: evolve_pass<R, 24, SIGN, OP>(sm, g, table); break;
    case 32: evolve_pass<R, 32, SIGN, OP>(sm, g, table); break;
    default: evolve_pass<R, 48, SIGN, OP>(sm, g, table); break;
  }
}

// in = out: psi <- transform back [ factor . transform_SIGN [psi] ].
// INIT: out = (1 + the same of in) / V.
template <typename R, int SIGN, int OP, bool INIT>
__global__ void __launch_bounds__(256) evolve_kernel(const cplx<R>* in, cplx<R>* out, int X, int Y, int Z,
                                                     const double* __restrict__ table) {
  extern __shared__ __align__(16) unsigned char evsm[];
  cplx<R>* sm = reinterpret_cast<cplx<R>*>(evsm);
  const int vol = X * Y * Z, zp = Z + 1;
  const cplx<R>* src = in + (size_t)blockIdx.x * vol;
  cplx<R>* dst = out + (size_t)blockIdx.x * vol;
  for (int e = threadIdx.x; e < vol; e += blockDim.x) {
    const int r = e / Z;
    sm[r * zp + (e - r * Z)] = src[e];
  }
  __syncthreads();
  const EvolvePass gz{X * Y, 1, zp, 1, 0}, gy{X * Z, Z, Y * zp, zp, 0}, gx{Y * Z, Z, zp, Y * zp, Y * Z};
  evolve_axis<R, SIGN, EV_NONE>(Z, sm, gz, nullptr);
  evolve_axis<R, SIGN, EV_NONE>(Y, sm, gy, nullptr);
  evolve_axis<R, SIGN, OP>(X, sm, gx, table);
  evolve_axis<R, -SIGN, EV_NONE>(Y, sm, gy, nullptr);
  evolve_axis<R, -SIGN, EV_NONE>(Z, sm, gz, nullptr);
  for (int e = threadIdx.x; e < vol; e += blockDim.x) {
    const int r = e / Z;
    cplx<R> v = sm[r * zp + (e - r * Z)];
    if constexpr (INIT) v = cplx<R>{(v.re + (R)1) / (R)vol, v.im / (R)vol};
    dst[e] = v;
  }
}

constexpr size_t kEvolveSmem = 227 * 1024;
size_t evolve_smem(size_t esz, const int d[3]) { return esz * (size_t)d[0] * d[1] * (d[2] + 1); }

template <typename R, int SIGN, int OP, bool INIT>
nrcps_status launch_evolve(nrcps_context* ctx, const void* in, void* out, int batch, const int d[3],
                           const double* table) {
  const size_t smem = evolve_smem(sizeof(cplx<R>), d);
  auto kern = evolve_kernel<R, SIGN, OP, INIT>;
  NRCPS_TRY(allow_smem(ctx, (const void*)kern, kEvolveSmem, "evolve: smem attribute"));
  // a thread per pencil of the axis with the most, at most 256
  int most = d[0] * d[1] > d[0] * d[2] ? d[0] * d[1] : d[0] * d[2];
  if (d[1] * d[2] > most) most = d[1] * d[2];
  const int threads = most >= 256 ? 256 : (most + 31) / 32 * 32;
  kern<<<(unsigned)batch, threads, smem, ctx->stream>>>(reinterpret_cast<const cplx<R>*>(in),
                                                        reinterpret_cast<cplx<R>*>(out), d[0], d[1], d[2], table);
  ctx->launches++;
  return check_launch(ctx, "evolve_kernel");
}

}  // namespace

// Whether one orbital of these extents fits a CTA's shared memory.
bool evolve_fits(nrcps_precision prec, const int d[3]) {
  return evolve_smem(prec == NRCPS_F64 ? sizeof(cplx<double>) : sizeof(cplx<float>), d) <= kEvolveSmem;
}

// psi <- B[w . F[psi]] with w complex (interleaved FP64) or real (FP64).
nrcps_status evolve_step(nrcps_context* ctx, void* psi, int batch, const int d[3], const double* w, bool w_complex,
                         nrcps_precision prec) {
  if (prec == NRCPS_F64)
    return w_complex ? launch_evolve<double, -1, EV_COMPLEX, false>(ctx, psi, psi, batch, d, w)
                     : launch_evolve<double, -1, EV_REAL, false>(ctx, psi, psi, batch, d, w);
  return w_complex ? launch_evolve<float, -1, EV_COMPLEX, false>(ctx, psi, psi, batch, d, w)
                   : launch_evolve<float, -1, EV_REAL, false>(ctx, psi, psi, batch, d, w);
}

// fld <- (1 + F[c . B[phi]]) / V, FP64.
nrcps_status evolve_initialize(nrcps_context* ctx, const double* phi, const double* c, const int d[3], double* fld) {
  return launch_evolve<double, +1, EV_REAL, true>(ctx, phi, fld, 1, d, c);
}

}  // namespace nrcps

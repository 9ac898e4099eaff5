// fused_one.cu -- the fused transfer-matrix step at L = 16 with a whole orbital
// in one CTA's shared memory.
//
//   psi(p) <- k(p) . B[ w(x) . F[ k(p) . psi(p) ] ]
//
// The passes are those of the cluster kernels (fused_step.cu) operation by
// operation, so the results are the same bit for bit; with the orbital in one
// CTA the x pass is a shared-memory pass like the others, and the cluster
// barriers and the remote loads and stores are gone.  Element (x, y, z) sits at
// (x L + y)(L + 1) + z: rows along z start four banks apart.
// Per orbital: y pencils from L2 (the next orbital is prefetched there
// meanwhile) times k(p); z; x, w, x back; z; y times k(p), streaming stores.
// A thread's last pencils of one orbital and its first of the next are the same
// columns, so four barriers per orbital do.  Nothing waits on another CTA.
//
// Three CTAs (FP64, 70 KB each; FP32: six) share an SM, two pencils per thread
// and pass, so that one's loads run beside the others' transforms.  FP64, 3500
// orbitals: 131 us (3500 GB/s of their one read and one write) against 161 for
// the pairs of CTAs (kind 0, cluster 2); Gaussian field 157 against 181; with a
// trap 144 against 176.  FP32, 14000 orbitals: 248 us against 270 (kind 4, the
// fastest variant at that size), 2100 orbitals 42 against 49.  At L = 24 an
// FP64 orbital fills the SM, its loads meet no other work, and the cluster of
// four is faster (627 orbitals, Gaussian: 166 against 150 us).
#include "fused.cuh"

namespace nrcps {

namespace {

template <typename R>
struct OneShape {
  static constexpr int L = 16, LP = L + 1, PLANE = L * LP;
  static constexpr size_t SMEM = sizeof(cplx<R>) * (size_t)L * PLANE;
  static constexpr int CTAS = sizeof(R) == 8 ? 3 : 6;
  static constexpr int THREADS = L * L / 2;  // two pencils per thread and pass
  static_assert(THREADS % 32 == 0, "whole warps");
  static_assert(CTAS * (SMEM + 1024) <= 228 * 1024, "the CTAs of an SM");
};

// FK: 1 Z2 bits (with or without a position factor), 2 any other field.
template <typename R, int FK>
__global__ void __launch_bounds__(OneShape<R>::THREADS, OneShape<R>::CTAS) fused_step_one_kernel(FusedArgs f) {
  using Sh = OneShape<R>;
  typedef typename vec2<R>::type V2;
  constexpr int L = Sh::L, V = L * L * L, LP = Sh::LP, PLANE = Sh::PLANE;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  cplx<R>* sm = reinterpret_cast<cplx<R>*>(smem_raw);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  R wp_hi, wp_lo, wm_hi, wm_lo;
  split<R>(f.w_plus, wp_hi, wp_lo);
  split<R>(f.w_minus, wm_hi, wm_lo);
  const bool w_exact = wp_lo == (R)0 && wm_lo == (R)0;
  for (long orb = blockIdx.x; orb < f.n_orb_total; orb += gridDim.x) {
    const long conf = orb / f.batch;
    const uint64_t kb = f.off0 + (f.conf_base ? __ldg(f.conf_base + conf) : (uint64_t)conf * f.conf_stride);
    cplx<R>* gpsi = reinterpret_cast<cplx<R>*>(f.psi) + (size_t)orb * V;
    if (lane == 0 && orb + gridDim.x < f.n_orb_total) {
      constexpr int SHARE = V / (Sh::THREADS / 32);
      static_assert(V % (Sh::THREADS / 32) == 0 && SHARE * sizeof(cplx<R>) % 16 == 0, "equal shares of 16-byte units");
      prefetch_l2(gpsi + (size_t)gridDim.x * V + (size_t)warp * SHARE, SHARE * (uint32_t)sizeof(cplx<R>));
    }
    cplx<R> x[L];
    // ---- times k(p), forward along y: pencil (x, z)
#pragma unroll 1
    for (int p = tid; p < L * L; p += Sh::THREADS) {
      const int z = p % L, xx = p / L, site0 = xx * L * L + z;
#pragma unroll
      for (int y = 0; y < L; ++y) {
        const V2 t = __ldcg(reinterpret_cast<const V2*>(gpsi) + site0 + y * L);
        x[y] = cplx<R>{t.x, t.y};
      }
#pragma unroll
      for (int y = 0; y < L; ++y) x[y] = apply_kin<R>(f, site0 + y * L, x[y]);
      fft::dft<L, -1, R, false>(x);
      cplx<R>* col = sm + xx * PLANE + z;
#pragma unroll
      for (int y = 0; y < L; ++y) col[y * LP] = x[y];
    }
    __syncthreads();
    // ---- forward along z in place: pencil (x, y)
#pragma unroll 1
    for (int p = tid; p < L * L; p += Sh::THREADS) {
      cplx<R>* row = sm + p * LP;
#pragma unroll
      for (int j = 0; j < L; ++j) x[j] = row[j];
      fft::dft<L, -1, R, false>(x);
#pragma unroll
      for (int j = 0; j < L; ++j) row[j] = x[j];
    }
    __syncthreads();
    // ---- along x, times w, and back: pencil (y, z)
#pragma unroll 1
    for (int p = tid; p < L * L; p += Sh::THREADS) {
      cplx<R>* col = sm + p / L * LP + p % L;
#pragma unroll
      for (int xx = 0; xx < L; ++xx) x[xx] = col[xx * PLANE];
      fft::dft<L, -1, R, false>(x);
      if constexpr (FK == 1) {
        const uint64_t k0 = kb + (uint64_t)p;
        const uint32_t* words = reinterpret_cast<const uint32_t*>(f.field) + (k0 >> 5);
        const int bit = (int)(k0 & 31);
        if (f.zpos) {
          constexpr int CH = 4;  // words and weights of four sites ahead of their use
#pragma unroll
          for (int x0 = 0; x0 < L; x0 += CH) {
            uint32_t word[CH];
            typename ZposEntry<R>::type w[CH];
#pragma unroll
            for (int i = 0; i < CH; ++i) {
              word[i] = __ldg(words + (x0 + i) * (L * L / 32));
              w[i] = __ldg(reinterpret_cast<const typename ZposEntry<R>::type*>(f.zpos) + p + (x0 + i) * L * L);
            }
#pragma unroll
            for (int i = 0; i < CH; ++i) x[x0 + i] = scale_w_entry<R, false>(w[i], (word[i] >> bit) & 1u, x[x0 + i]);
          }
        } else if (w_exact) {
#pragma unroll
          for (int xx = 0; xx < L; ++xx) {
            const bool up = (__ldg(words + xx * (L * L / 32)) >> bit) & 1u;
            x[xx] = scale_w1<R, false>(x[xx], up ? wp_hi : wm_hi);
          }
        } else {
#pragma unroll
          for (int xx = 0; xx < L; ++xx) {
            const bool up = (__ldg(words + xx * (L * L / 32)) >> bit) & 1u;
            x[xx] = scale_w<R, false>(x[xx], up ? wp_hi : wm_hi, up ? wp_lo : wm_lo);
          }
        }
      } else {
        apply_w_pencil<R, L, L * L>(f, kb, p, x);
      }
      fft::dft<L, +1, R, false>(x);
#pragma unroll
      for (int xx = 0; xx < L; ++xx) col[xx * PLANE] = x[xx];
    }
    __syncthreads();
    // ---- backward along z
#pragma unroll 1
    for (int p = tid; p < L * L; p += Sh::THREADS) {
      cplx<R>* row = sm + p * LP;
#pragma unroll
      for (int j = 0; j < L; ++j) x[j] = row[j];
      fft::dft<L, +1, R, false>(x);
#pragma unroll
      for (int j = 0; j < L; ++j) row[j] = x[j];
    }
    __syncthreads();
    // ---- backward along y, times k(p)
#pragma unroll 1
    for (int p = tid; p < L * L; p += Sh::THREADS) {
      const int z = p % L, xx = p / L, site0 = xx * L * L + z;
      const cplx<R>* col = sm + xx * PLANE + z;
#pragma unroll
      for (int y = 0; y < L; ++y) x[y] = col[y * LP];
      fft::dft<L, +1, R, false>(x);
#pragma unroll
      for (int y = 0; y < L; ++y) {
        const cplx<R> v = apply_kin<R>(f, site0 + y * L, x[y]);
        __stcs(reinterpret_cast<V2*>(gpsi) + site0 + y * L, V2{v.re, v.im});
      }
    }
  }
}

template <typename R>
nrcps_status launch_one(nrcps_context* ctx, const FusedArgs& f) {
  using Sh = OneShape<R>;
  const bool z2 = f.field_mode == 1 && (f.pos == nullptr || f.zpos != nullptr);
  void (*kern)(FusedArgs) = z2 ? fused_step_one_kernel<R, 1> : fused_step_one_kernel<R, 2>;
  NRCPS_TRY(allow_smem(ctx, (const void*)kern, Sh::SMEM, "fused_step_one: smem attribute"));
  const long slots = (long)ctx->sm_count * Sh::CTAS;
  const long grid = f.n_orb_total < slots ? f.n_orb_total : slots;
  kern<<<(unsigned)grid, Sh::THREADS, Sh::SMEM, ctx->stream>>>(f);
  ctx->launches++;
  return check_launch(ctx, "fused_step_one_kernel");
}

}  // namespace

// Orbitals that are in flight at a time, 0 where no kernel exists.
int fused_one_slots(const nrcps_context* ctx, nrcps_precision prec, int L) {
  if (L != 16) return 0;
  return ctx->sm_count * (prec == NRCPS_F64 ? OneShape<double>::CTAS : OneShape<float>::CTAS);
}

nrcps_status fused_one_step(nrcps_context* ctx, nrcps_precision prec, const FusedArgs& f) {
  return prec == NRCPS_F64 ? launch_one<double>(ctx, f) : launch_one<float>(ctx, f);
}

}  // namespace nrcps

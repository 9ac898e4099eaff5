// fused_park.cu -- the fused transfer-matrix step of FP32 orbitals at L = 32
// with the whole orbital inside one SM.
//
//   psi(p) <- k(p) . B[ w(x) . F[ k(p) . psi(p) ] ]
//
// An orbital of 32^3 complex floats is 256 KB, more than the 227 KB of shared
// memory, which is why the cluster kernels (fused_step.cu) spread it over
// eight CTAs and run the x pass through the peers' shared memory.  Here one
// CTA of 16 warps holds it alone: the x transform is split by the parity of
// p_x, one half of the orbital (16 x-planes) sits in shared memory at a time
// and the other is parked in tensor memory (one 256-column allocation, 64
// words per thread, read and written by the thread that owns the pencil).
// Nothing crosses between SMs.
//
// What bounds it: 19456 orbitals take 3.54 ms (2880 GB/s of the orbitals' one
// read and one write, 0.44 of a copy; kind 11 on clusters of 8: 4.78 ms).  Of
// the cluster kernel's 4.78 ms the exchange through distributed shared memory
// was 0.75 (with the x pass read from a CTA's own memory instead: 4.03), and
// its data movement alone, without any transform, took 3.99.  Here the FMA
// pipe is busy 50 % and an instruction issues in 58 % of the cycles; an
// orbital takes about 51 k cycles of an SM: 27 k of FMA work, 19 k of
// shared-memory accesses, which overlap in part only, and 8 k of exposed
// loads and stores.  Hence: rows pass through a staging buffer by cp.async
// ahead of use and leave by bulk copy (loads and stores by the threads
// themselves instead: 4.08 ms), and half of k(p) stays in tensor memory.
// Staging 16 or 12 of a plane's 32 rows instead of 22 (all that fit): 3.65,
// 3.61 ms; the next orbital not prefetched into L2: 3.63; mbarriers instead of
// the block barriers ahead of the buffer reuses: 3.64.
//
// Per orbital, half h = p_x mod 2 (plane m of a half is p_x = 2 m + h):
//   1. h = 0, 1: warp m transforms plane m alone: y pencils from L2 (lane =
//      z, times k(p)), into its 8 KB plane of shared memory, z pencils in
//      place (lane = y); no block barrier in between;
//      h = 0: thread (z, y) and (z, y + 16) takes its two half pencils along
//      x, transforms them (the even half of the radix-4 stage) and parks
//      the 16 results of each;
//   2. h = 1 in shared memory: the odd half of the x transform, the last
//      butterflies with the parked half, times w, the inverse transform
//      along x; the odd outputs go back to shared memory, the even ones to
//      tensor memory;
//   3. h = 1, then h = 0 (from tensor memory into shared memory): inverse
//      along z and y, times k(p), streaming stores.
// The transforms are those of the cluster kernels operation by operation
// (fft::Dft<32>: its even and odd halves meet only in the last radix-4
// stage), so the results are the same bit for bit.
#include "fused.cuh"

namespace nrcps {

namespace {

constexpr int PL = 32;                  // lattice extent
constexpr int PH = PL / 2;              // planes per half
constexpr int PLD = PL + 1;             // padded z row
constexpr int PPLANE = PL * PLD;        // elements per plane
constexpr int PTHREADS = PH * PL;       // one warp per plane
constexpr uint32_t PCOLS = 512;         // tensor memory columns: per lane quarter 4 warps x (64 parked + 64 k(p)) words
constexpr uint32_t PKCOL = 256;         // first column of k(p)
constexpr int PSROWS = 22;              // rows of a plane that pass through the warp's staging buffer
constexpr size_t PSMEM = sizeof(float2) * ((size_t)PH * PPLANE + (size_t)PH * PSROWS * PL) + 16;

typedef cplx<float> cf;

// 32 words of this thread's lane, columns addr .. addr + 31
__device__ __forceinline__ void park_store(uint32_t addr, const cf* v) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};" ::"r"(addr),
      "f"(v[0].re), "f"(v[0].im), "f"(v[1].re), "f"(v[1].im), "f"(v[2].re), "f"(v[2].im), "f"(v[3].re), "f"(v[3].im),
      "f"(v[4].re), "f"(v[4].im), "f"(v[5].re), "f"(v[5].im), "f"(v[6].re), "f"(v[6].im), "f"(v[7].re), "f"(v[7].im),
      "f"(v[8].re), "f"(v[8].im), "f"(v[9].re), "f"(v[9].im), "f"(v[10].re), "f"(v[10].im), "f"(v[11].re),
      "f"(v[11].im), "f"(v[12].re), "f"(v[12].im), "f"(v[13].re), "f"(v[13].im), "f"(v[14].re), "f"(v[14].im),
      "f"(v[15].re), "f"(v[15].im)
      : "memory");
}
__device__ __forceinline__ void park_store_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// ... read back; the wait is part of the statement, so no use of the values can move ahead of it
__device__ __forceinline__ void park_load(uint32_t addr, cf* v) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];\n"
      "tcgen05.wait::ld.sync.aligned;"
      : "=f"(v[0].re), "=f"(v[0].im), "=f"(v[1].re), "=f"(v[1].im), "=f"(v[2].re), "=f"(v[2].im), "=f"(v[3].re),
        "=f"(v[3].im), "=f"(v[4].re), "=f"(v[4].im), "=f"(v[5].re), "=f"(v[5].im), "=f"(v[6].re), "=f"(v[6].im),
        "=f"(v[7].re), "=f"(v[7].im), "=f"(v[8].re), "=f"(v[8].im), "=f"(v[9].re), "=f"(v[9].im), "=f"(v[10].re),
        "=f"(v[10].im), "=f"(v[11].re), "=f"(v[11].im), "=f"(v[12].re), "=f"(v[12].im), "=f"(v[13].re),
        "=f"(v[13].im), "=f"(v[14].re), "=f"(v[14].im), "=f"(v[15].re), "=f"(v[15].im)
      : "r"(addr)
      : "memory");
}

// The half of fft::Dft<32, -1> that takes the inputs of parity H: on entry
// v[m] = x[2 m + H]; on exit v[k] and v[k + 8] (k < 8) hold the sum and the
// difference of its two radix-4 inputs of output k (the difference of the
// odd half times -i).
template <int H>
__device__ __forceinline__ void half_forward(cf* v) {
  cf a[8], b[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    a[j] = v[2 * j];
    b[j] = v[2 * j + 1];
  }
  fft::Dft<8, -1, float>::run(a);
  fft::Dft<8, -1, float>::run(b);
  fft::static_for<8>([&](auto kc) {
    constexpr int k = decltype(kc)::value;
    const cf ta = fft::twiddle<32, H * k, -1, float>(a[k]), tb = fft::twiddle<32, (H + 2) * k, -1, float>(b[k]);
    v[k] = fft::add(ta, tb);
    v[k + 8] = fft::sub(ta, tb);
    if constexpr (H == 1) v[k + 8] = fft::mul_i<-1>(v[k + 8]);
  });
}

// 32 x 32 bits across a warp: lane i's bit j becomes lane j's bit i
__device__ __forceinline__ uint32_t transpose_bits(uint32_t v, int lane) {
  uint32_t m = 0x0000FFFFu;
#pragma unroll
  for (int s = 16; s > 0; s >>= 1) {
    const uint32_t o = __shfl_xor_sync(0xffffffffu, v, s);
    v = (lane & s) ? ((v & ~m) | ((o >> s) & m)) : ((v & m) | ((o & m) << s));
    m ^= m << (s >> 1);
  }
  return v;
}

// FK as in fused_step_async_kernel: 1 Z2 bits (with or without a position
// factor), 2 any other field, 3 a real FP32 weight table.
template <int FK>
__global__ void __launch_bounds__(PTHREADS, 1) fused_step_park_kernel(FusedArgs f) {
  constexpr int V = PL * PL * PL;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  cf* sm = reinterpret_cast<cf*>(smem_raw);
  uint32_t* slot = reinterpret_cast<uint32_t*>(sm + PH * PPLANE + PH * PSROWS * PL);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     (uint32_t)__cvta_generic_to_shared(slot)),
                 "r"(PCOLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  // a warp reaches the 32 lanes of its quarter (warp mod 4)
  const uint32_t tmem = *slot;
  const uint32_t park = tmem + ((uint32_t)(warp & 3) << 21) + (uint32_t)(warp >> 2) * 64;

  float wp_hi, wp_lo, wm_hi, wm_lo;
  split<float>(f.w_plus, wp_hi, wp_lo);
  split<float>(f.w_minus, wm_hi, wm_lo);
  const bool w_exact = wp_lo == 0.f && wm_lo == 0.f;
  cf* plane = sm + warp * PPLANE;  // this warp's plane of the half in shared memory
  cf* stage = sm + PH * PPLANE + warp * PSROWS * PL;  // and its staging rows
  const float2* kin0 = f.kin_f + 2 * warp * PL * PL + lane;  // k(p) of (p_x = 2 warp, y = 0, z = lane)
  const uint32_t kpark = park + PKCOL;
  // k(p) of this warp's odd plane stays in tensor memory
#pragma unroll 1
  for (int c = 0; c < 2; ++c) {
    cf k[PH];
#pragma unroll
    for (int y = 0; y < PH; ++y) {
      const float2 t = __ldg(kin0 + PL * PL + (c * PH + y) * PL);
      k[y] = cf{t.x, t.y};
    }
    park_store(kpark + 32 * c, k);
  }
  park_store_wait();
  auto scale_even = [&](cf* x) {
#pragma unroll
    for (int y = 0; y < PL; ++y) {
      const float2 k = __ldg(kin0 + y * PL);
      x[y] = scale2<float>(x[y], k.x, k.y);
    }
  };
  auto scale_odd = [&](cf* x) {
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      cf k[PH];
      park_load(kpark + 32 * c, k);
#pragma unroll
      for (int y = 0; y < PH; ++y) x[c * PH + y] = scale2<float>(x[c * PH + y], k[y].re, k[y].im);
    }
  };
  // the first rows of one of this warp's planes on their way into its staging
  // rows, 16 bytes per lane and copy
  auto fetch = [&](const float2* p) {
    const char* src = reinterpret_cast<const char*>(p) + 16 * lane;
    const uint32_t dst = (uint32_t)__cvta_generic_to_shared(stage) + 16 * lane;
#pragma unroll
    for (int i = 0; i < PSROWS / 2; ++i)
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + 512 * i), "l"(src + 512 * i) : "memory");
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  // rows in shared memory on their way to HBM (written by the whole warp before)
  auto send = [&](float2* dst, const cf* src, uint32_t bytes) {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncwarp();
    if (lane == 0) {
      asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst),
                   "r"((uint32_t)__cvta_generic_to_shared(src)), "r"(bytes)
                   : "memory");
      asm volatile("cp.async.bulk.commit_group;" ::: "memory");
    }
  };
  auto sent = [&]() {  // ... have left it
    if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
    __syncwarp();
  };
  long orb = blockIdx.x;
  if (orb < f.n_orb_total) fetch(reinterpret_cast<float2*>(f.psi) + (size_t)orb * V + 2 * warp * PL * PL);

  for (; orb < f.n_orb_total; orb += gridDim.x) {
    const long conf = orb / f.batch;
    const uint64_t kb = f.off0 + (f.conf_base ? __ldg(f.conf_base + conf) : (uint64_t)conf * f.conf_stride);
    float2* gpsi = reinterpret_cast<float2*>(f.psi) + (size_t)orb * V;
    // the next orbital on its way into L2 meanwhile, 16 KB per warp
    if (lane == 0 && orb + gridDim.x < f.n_orb_total)
      prefetch_l2(gpsi + (size_t)gridDim.x * V + (size_t)warp * (V / PH), V / PH * 8);
    // Z2: the sign words of rows (x = lane, y = warp and warp + 16), turned
    // into one word of x signs per z further down
    uint32_t up[2] = {0, 0};
    if constexpr (FK == 1) {
      const uint32_t* words = reinterpret_cast<const uint32_t*>(f.field) + (kb >> 5);
      const int sh = (int)(kb & 31);
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const int row = lane * PL + warp + PH * q;
        const uint32_t lo = __ldg(words + row);
        up[q] = sh ? __funnelshift_r(lo, __ldg(words + row + 1), sh) : lo;
      }
    }
    cf x[PL];
    const float2* even = gpsi + 2 * warp * PL * PL + lane;
#pragma unroll
    for (int y = PSROWS; y < PL; ++y) {
      const float2 t = __ldcg(even + y * PL);
      x[y] = cf{t.x, t.y};
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncwarp();
#pragma unroll
    for (int y = 0; y < PSROWS; ++y) x[y] = stage[y * PL + lane];
    __syncwarp();
    fetch(gpsi + (2 * warp + 1) * PL * PL);
    scale_even(x);
    // ---- forward along y and z, plane by plane, then along x
#pragma unroll 1
    for (int h = 0; h < 2; ++h) {
      fft::Dft<PL, -1, float>::run(x);
      if (h) __syncthreads();  // the even half has been read out of shared memory
      else sent();             // the previous orbital's even plane has left
#pragma unroll
      for (int y = 0; y < PL; ++y) plane[y * PLD + lane] = x[y];
      __syncwarp();
      cf* row = plane + lane * PLD;
#pragma unroll
      for (int j = 0; j < PL; ++j) x[j] = row[j];
      fft::Dft<PL, -1, float>::run(x);
#pragma unroll
      for (int j = 0; j < PL; ++j) row[j] = x[j];
      __syncthreads();
      if (h == 0) {
        const float2* odd = even + PL * PL;
#pragma unroll
        for (int y = PSROWS; y < PL; ++y) {
          const float2 t = __ldcg(odd + y * PL);
          x[y] = cf{t.x, t.y};
        }
#pragma unroll 1
        for (int q = 0; q < 2; ++q) {
          const cf* col = sm + (warp + PH * q) * PLD + lane;
          cf v[PH];
#pragma unroll
          for (int m = 0; m < PH; ++m) v[m] = col[m * PPLANE];
          half_forward<0>(v);
          park_store(park + 32 * q, v);
        }
        park_store_wait();
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncwarp();
#pragma unroll
        for (int y = 0; y < PSROWS; ++y) x[y] = stage[y * PL + lane];
        scale_odd(x);
      }
    }
    if constexpr (FK == 1) {
      up[0] = transpose_bits(up[0], lane);
      up[1] = transpose_bits(up[1], lane);
    }
    // ---- along x: the last butterflies, times w, and back
#pragma unroll 1
    for (int q = 0; q < 2; ++q) {
      const int y = warp + PH * q;
      const int site0 = y * PL + lane;  // site of x = 0
      cf* col = sm + y * PLD + lane;
      {
        cf o[PH], e[PH];
#pragma unroll
        for (int m = 0; m < PH; ++m) o[m] = col[m * PPLANE];
        half_forward<1>(o);
        park_load(park + 32 * q, e);
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          x[k] = fft::add(e[k], o[k]);
          x[k + 16] = fft::sub(e[k], o[k]);
          x[k + 8] = fft::add(e[k + 8], o[k + 8]);
          x[k + 24] = fft::sub(e[k + 8], o[k + 8]);
        }
      }
      if constexpr (FK == 1) {
        const uint32_t s = up[q];
        if (f.zpos) {
#pragma unroll
          for (int xx = 0; xx < PL; ++xx)
            x[xx] = scale_w_zpos<float, false>(f.zpos, site0 + xx * PL * PL, (s >> xx) & 1u, x[xx]);
        } else if (w_exact) {
#pragma unroll
          for (int xx = 0; xx < PL; ++xx) x[xx] = scale_w1<float, false>(x[xx], ((s >> xx) & 1u) ? wp_hi : wm_hi);
        } else {
#pragma unroll
          for (int xx = 0; xx < PL; ++xx) {
            const bool u = (s >> xx) & 1u;
            x[xx] = scale_w<float, false>(x[xx], u ? wp_hi : wm_hi, u ? wp_lo : wm_lo);
          }
        }
      } else if constexpr (FK == 3) {
        const float* tab = reinterpret_cast<const float*>(f.field) + kb + site0;
#pragma unroll
        for (int xx = 0; xx < PL; ++xx) {
          const float w = __ldg(tab + xx * PL * PL);
          x[xx] = cf{__fmul_rn(x[xx].re, w), __fmul_rn(x[xx].im, w)};
        }
      } else {
        apply_w_pencil<float, PL, PL * PL>(f, kb, site0, x);
      }
      fft::Dft<PL, +1, float>::run(x);
      cf e[PH];
#pragma unroll
      for (int m = 0; m < PH; ++m) {
        e[m] = x[2 * m];
        col[m * PPLANE] = x[2 * m + 1];
      }
      park_store(park + 32 * q, e);
    }
    park_store_wait();
    __syncthreads();
    // ---- backward along z and y: the odd half, then the parked one
#pragma unroll 1
    for (int h = 1; h >= 0; --h) {
      cf* row = plane + lane * PLD;
#pragma unroll
      for (int j = 0; j < PL; ++j) x[j] = row[j];
      fft::Dft<PL, +1, float>::run(x);
#pragma unroll
      for (int j = 0; j < PL; ++j) row[j] = x[j];
      __syncwarp();
      if (h == 0 && orb + gridDim.x < f.n_orb_total) {
        sent();  // the odd plane has left the staging rows: the next orbital's even plane may land there
        fetch(gpsi + (size_t)gridDim.x * V + 2 * warp * PL * PL);
      }
#pragma unroll
      for (int y = 0; y < PL; ++y) x[y] = plane[y * PLD + lane];
      fft::Dft<PL, +1, float>::run(x);
      float2* out = gpsi + (2 * warp + h) * PL * PL;
      if (h) {
        scale_odd(x);
#pragma unroll
        for (int y = 0; y < PSROWS; ++y) stage[y * PL + lane] = x[y];
        send(out, stage, PSROWS * PL * sizeof(cf));
#pragma unroll
        for (int y = PSROWS; y < PL; ++y) __stcs(out + y * PL + lane, make_float2(x[y].re, x[y].im));
      } else {
        scale_even(x);
        __syncwarp();
#pragma unroll
        for (int y = 0; y < PL; ++y) plane[y * PL + lane] = x[y];
        send(out, plane, PL * PL * sizeof(cf));
      }
      if (h) {
        __syncthreads();  // every warp has read its odd plane
#pragma unroll 1
        for (int q = 0; q < 2; ++q) {
          cf e[PH];
          park_load(park + 32 * q, e);
          cf* col = sm + (warp + PH * q) * PLD + lane;
#pragma unroll
          for (int m = 0; m < PH; ++m) col[m * PPLANE] = e[m];
        }
        __syncthreads();
      }
    }
  }
  if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(PCOLS) : "memory");
}

}  // namespace

// One step of n_orb_total FP32 orbitals at L = 32 (arguments as fused_step
// fills them).
nrcps_status fused_park_step(nrcps_context* ctx, const FusedArgs& f) {
  const bool z2 = f.field_mode == 1 && (f.pos == nullptr || f.zpos != nullptr);
  void (*kern)(FusedArgs) = z2                  ? fused_step_park_kernel<1>
                            : f.field_mode == 3 ? fused_step_park_kernel<3>
                                                : fused_step_park_kernel<2>;
  NRCPS_TRY(allow_smem(ctx, (const void*)kern, PSMEM, "fused_step_park: smem attribute"));
  const long grid = f.n_orb_total < ctx->sm_count ? f.n_orb_total : ctx->sm_count;
  kern<<<(unsigned)grid, PTHREADS, PSMEM, ctx->stream>>>(f);
  ctx->launches++;
  return check_launch(ctx, "fused_step_park_kernel");
}

}  // namespace nrcps

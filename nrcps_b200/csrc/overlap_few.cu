// overlap_few.cu -- the Slater overlap of FP32 orbitals with up to ten dense
// sources on the CUDA cores
//
//   S[c][s][t] = sum_p conj(src_s(p)) psi_{c,t}(p)
//
// (OneBody::Project, src/one_body/noarch/one_body_project.C:14-27, into
// SlaterDet's S, src/slater_det/slater_det.C:33-37.)
//
// With ten sources the tensor-core kernel (overlap_tc.cu) fills 20 of the 64
// rows of its source operand and is bound by shared memory: an orbital tile is
// split into TF32 halves there and read back by the tensor core, 144 KB of
// traffic for 16 KB of orbitals.  Here the operands are plain FP32 (the sources
// rounded once, 24 bits against the 22 of a TF32 pair) and each is read once
// per block of five.  One cluster of up to eight CTAs per configuration and ten
// orbitals, CTA r takes every C-th tile of 128 sites; tiles come in by cp.async,
// three stages; a warp owns a 5 x 5 block (fewer blocks: several warps each),
// a lane one site at a time.  Products as in pair_sym.cu: P += a . b,
// Q += a . swap(b), packed, re S = P.x + P.y, im S = Q.x - Q.y; after 32 sites
// the warp's lanes sum up by a reduce-scatter, then FP64.
//
// At L = 48, n = 10, 128 configurations: 459 us (2470 GB/s; the tensor-core kernel
// 496) at an error against 64 bits of 1.3e-7 (6.4e-7).  The FMA pipe is busy 51
// % of the cycles, a warp waits most for its own last FMA: 168 registers leave
// twelve warps per SM.
#include <cooperative_groups.h>

#include "lane_sums.cuh"

namespace nrcps {
namespace cg = cooperative_groups;

namespace {

constexpr int FB = 5;       // rows of a block
constexpr int FT = 128;     // sites of a tile
constexpr int FUNITS = FT / 32;
constexpr int FSTAGES = 3;
constexpr int FFLUSH = 32;  // sites of one FP32 sum
constexpr int FWARPS = 4, FTHREADS = 32 * FWARPS, FCTAS = 3;

template <int NS, int NT>  // blocks of sources and orbitals, 1 or 2 each
struct FewShape {
  static constexpr int ROWS = FB * (NS + NT), GROUPS = FWARPS / (NS * NT);
  static constexpr size_t STAGE = sizeof(float2) * ROWS * FT;
  static constexpr size_t SMEM = FSTAGES * STAGE;
  static_assert(sizeof(double) * 64 * FWARPS <= SMEM, "the final sums lie over the stages");
};

__device__ __forceinline__ void copy16(void* dst, const void* src, bool take) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src),
               "r"(take ? 16 : 0)
               : "memory");
}

// vol even, src and psi on 16 bytes
template <int NS, int NT>
__global__ void __launch_bounds__(FTHREADS, FCTAS)
    overlap_few_kernel(const float2* __restrict__ src, int ns, const float2* __restrict__ psi, int nt, long vol,
                       double* __restrict__ S) {
  using Sh = FewShape<NS, NT>;
  extern __shared__ __align__(16) unsigned char fsm[];
  cg::cluster_group cluster = cg::this_cluster();
  const int split = (int)cluster.num_blocks(), rank = (int)cluster.block_rank();
  const long conf = blockIdx.x / split;
  const int t0 = (int)blockIdx.y * 2 * FB, nth = nt - t0 < 2 * FB ? nt - t0 : 2 * FB;  // this CTA's orbitals
  const float2* orb = psi + ((size_t)conf * nt + t0) * vol;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  auto stage = [&](int b) { return reinterpret_cast<float2*>(fsm + b * Sh::STAGE); };
  const long ntiles = (vol + FT - 1) / FT;
  const int rows = ns + nth;
  // padding rows stay zero: sources at [0, ns), orbitals from row FB NS on
  for (int r = warp; r < Sh::ROWS; r += FWARPS)
    if (r < FB * NS ? r >= ns : r - FB * NS >= nth)
      for (int e = lane; e < FSTAGES * FT; e += 32) stage(e / FT)[r * FT + e % FT] = make_float2(0.f, 0.f);
  auto issue = [&](int b, long tile) {
    if (tile < ntiles) {
      float2* x = stage(b);
      for (int r = warp; r < rows; r += FWARPS) {
        const float2* row = r < ns ? src + (size_t)r * vol : orb + (size_t)(r - ns) * vol;
        float2* to = x + (r < ns ? r : FB * NS + r - ns) * FT;
#pragma unroll
        for (int u = 0; u < FT / 64; ++u) {
          const int q = 64 * u + 2 * lane;
          const bool take = tile * FT + q < vol;
          copy16(to + q, row + (take ? tile * FT + q : 0), take);
        }
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  const int block = warp / Sh::GROUPS, unit0 = warp % Sh::GROUPS;
  const int bs = block / NT, bt = block % NT;
  float2 P[FB * FB], Q[FB * FB];
  double sum[2] = {0.0, 0.0};
  int count = 0;
  auto clear = [&]() {
#pragma unroll
    for (int e = 0; e < FB * FB; ++e) P[e] = Q[e] = make_float2(0.f, 0.f);
    count = 0;
  };
  auto flush = [&]() {
    float v[2 * FB * FB];
#pragma unroll
    for (int e = 0; e < FB * FB; ++e) {
      v[2 * e] = P[e].x + P[e].y;
      v[2 * e + 1] = Q[e].x - Q[e].y;
    }
    reduce_scatter<2 * FB * FB>(v, lane);
    sum[0] += (double)v[0];
    sum[1] += (double)v[1];
    clear();
  };
  clear();
#pragma unroll
  for (int b = 0; b < FSTAGES - 1; ++b) issue(b, rank + (long)b * split);
  int buf = 0;
  for (long tile = rank; tile < ntiles; tile += split) {
    asm volatile("cp.async.wait_group %0;" ::"n"(FSTAGES - 2) : "memory");
    __syncthreads();  // this tile is in, and every warp has left the one whose buffer comes next
    issue(buf == 0 ? FSTAGES - 1 : buf - 1, tile + (FSTAGES - 1) * (long)split);
    const float2* a = stage(buf) + bs * FB * FT + lane;
    const float2* b = stage(buf) + (FB * NS + bt * FB) * FT + lane;
#pragma unroll 1
    for (int u = unit0; u < FUNITS; u += Sh::GROUPS) {
      float2 y[FB], z[FB];
#pragma unroll
      for (int t = 0; t < FB; ++t) {
        y[t] = b[t * FT + 32 * u];
        z[t] = make_float2(y[t].y, y[t].x);
      }
#pragma unroll
      for (int s = 0; s < FB; ++s) {
        const float2 x = a[s * FT + 32 * u];
#pragma unroll
        for (int t = 0; t < FB; ++t) {
          P[s * FB + t] = __ffma2_rn(x, y[t], P[s * FB + t]);
          Q[s * FB + t] = __ffma2_rn(x, z[t], Q[s * FB + t]);
        }
      }
      if (++count == FFLUSH) flush();
    }
    buf = buf == FSTAGES - 1 ? 0 : buf + 1;
  }
  flush();
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  // every warp's sums over the stages, then the cluster's CTAs in rank order
  double* red = reinterpret_cast<double*>(fsm);  // [FWARPS][64]
  red[warp * 64 + 2 * lane] = sum[0];
  red[warp * 64 + 2 * lane + 1] = sum[1];
  cluster.sync();
  for (int e = rank * FTHREADS + threadIdx.x; e < 2 * ns * nth; e += split * FTHREADS) {
    const int c = e & 1, s = e / 2 / nth, t = e / 2 % nth;
    const int first = (s / FB * NT + t / FB) * Sh::GROUPS, k = 2 * (s % FB * FB + t % FB) + c;
    double v = 0.0;
    for (int r = 0; r < split; ++r) {
      const double* peer = cluster.map_shared_rank(red, r);
      for (int g = 0; g < Sh::GROUPS; ++g) v += peer[(first + g) * 64 + k];
    }
    S[2 * ((conf * ns + s) * (long)nt + t0 + t) + c] = v;
  }
  cluster.sync();  // peers keep their shared memory until every sum is read
}

__global__ void round_sources_kernel(const double2* __restrict__ src, long n, float2* __restrict__ out) {
  for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x)
    out[i] = make_float2((float)src[i].x, (float)src[i].y);
}

template <int NS, int NT>
nrcps_status launch_few(nrcps_context* ctx, const float* src, int ns, const void* psi, int nt, int nconf, long vol,
                        double* S) {
  using Sh = FewShape<NS, NT>;
  auto kern = overlap_few_kernel<NS, NT>;
  NRCPS_TRY(allow_smem(ctx, (const void*)kern, Sh::SMEM, "overlap_few: smem attribute"));
  // the split of a configuration that leaves the fewest rounds of CTAs per share
  const long groups = (nt + 2 * FB - 1) / (2 * FB), slots = (long)ctx->sm_count * FCTAS, ntiles = (vol + FT - 1) / FT;
  int split = 1;
  double best = 1e300;
  for (int s = 1; s <= 8 && s <= ntiles; ++s) {
    const double cost = (double)((nconf * groups * s + slots - 1) / slots) / s;
    if (cost < 0.97 * best) best = cost, split = s;
  }
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)split;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.gridDim = dim3((unsigned)((long)nconf * split), (unsigned)groups);
  cfg.blockDim = dim3(FTHREADS);
  cfg.dynamicSmemBytes = Sh::SMEM;
  cfg.stream = ctx->stream;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  ctx->launches++;
  return check_cuda(ctx, cudaLaunchKernelEx(&cfg, kern, reinterpret_cast<const float2*>(src), ns,
                                            reinterpret_cast<const float2*>(psi), nt, vol, S),
                    "overlap_few_kernel launch");
}

}  // namespace

// Where this kernel is the faster one (measured with ns = nt = N).  Small batches
// (128 MB of orbitals), where the tensor-core kernel's preparation and fill show:
// L = 32, ten orbitals, 33 configurations 46 against 89 us, 24 of seven at L = 8
// 15 against 22; but not those of very many configurations, which are a CTA each
// at least (L = 8, N = 2, 1000 of them 32 against 21), nor of one to three sources
// on many sites, where most of a block of five is padding (L = 48, N = 1, 100
// configurations 98 against 61), nor of one or two orbitals (L = 32, 10 sources, 200
// configurations 114 against 52), nor, with more than five, large volumes, where
// a cluster of eight per configuration leaves the chip empty (L = 48, N = 7, 16
// configurations 122 against 73).  Large ones where the blocks of five are full
// and a configuration has many tiles: L = 48, N = 10, 128 configurations 459
// against 496 (16: 135 against 114), L = 32, N = 5, 1000 350 against 517; N = 9 up
// to 128 configurations only (L = 32, 100 106 against 116, 500 486 against 442);
// not L = 48, N = 7, 180: 591 against 488, nor L = 16, N = 10, 4000: 670 against 531.
bool overlap_few_pays(int ns, int nt, int nconf, long vol) {
  if (ns > 2 * FB || nt > 65535L * 2 * FB) return false;  // (groups of orbitals are a grid's y)
  const long l32 = 32 * 32 * 32, sites = nconf * vol;
  if ((double)nt * sites <= (double)(1 << 24)) {
    if (ns <= 3) return nconf <= 128 && sites <= 1 << 22;
    if (nt <= 2) return nconf <= 128 && sites < 1 << 21;
    const long ctas = (long)nconf * ((nt + 2 * FB - 1) / (2 * FB));
    return ns <= FB ? ctas <= 512 : ctas <= 320 && vol <= l32;
  }
  const long padded = (long)((ns + FB - 1) / FB) * ((nt + FB - 1) / FB) * FB * FB, full = (long)ns * nt;
  return (9 * padded <= 10 * full || (4 * padded <= 5 * full && nconf <= 128)) && vol >= l32 &&
         (ns <= FB || vol == l32 || nconf >= 32);
}

// The sources as FP32 in `out` (8 ns vol bytes, on 16).
nrcps_status overlap_few_prepare(nrcps_context* ctx, const double* src, int ns, long vol, float* out) {
  const long n = (long)ns * vol;
  round_sources_kernel<<<grid_for(n, 256, (long)ctx->sm_count * 16), 256, 0, ctx->stream>>>(
      reinterpret_cast<const double2*>(src), n, reinterpret_cast<float2*>(out));
  ctx->launches++;
  return check_launch(ctx, "round_sources_kernel");
}

nrcps_status overlap_few(nrcps_context* ctx, const float* src, int ns, const void* psi, int nt, int nconf, long vol,
                         double* S) {
  if (ns <= FB)
    return nt <= FB ? launch_few<1, 1>(ctx, src, ns, psi, nt, nconf, vol, S)
                    : launch_few<1, 2>(ctx, src, ns, psi, nt, nconf, vol, S);
  return nt <= FB ? launch_few<2, 1>(ctx, src, ns, psi, nt, nconf, vol, S)
                  : launch_few<2, 2>(ctx, src, ns, psi, nt, nconf, vol, S);
}

}  // namespace nrcps

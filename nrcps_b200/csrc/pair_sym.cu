// pair_sym.cu -- pair matrices of one set of FP32 orbitals, 9 <= n <= 20
//
//   phi_st = sum_i w(i) psi_s(i) psi_t(opp(i)),  opp an involution, w even under it
//
// (TwoBody::Run, src/two_body/noarch/two_body_run.C:13-43, for the ensemble's
// pair sink.)  The sites pair up: with x = psi(i), y = psi(opp(i)), a pair
// adds w (x_s y_t + y_s x_t), symmetric in (s, t); a site that is its own
// partner adds the same with w/2.  Every orbital element is read once.
//
// One cluster of up to eight CTAs per configuration, CTA r takes every C-th
// tile of 128 sites i; tiles without a site i <= opp(i) are left out after a
// look at opp (bits in shared memory, a window of tiles at a time).  x and y
// of a tile's sites come in by cp.async, three stages; a warp owns one 5 x 5
// block of phi (on the diagonal the 15 entries of the triangle), a lane takes
// one pair of sites at a time.
//
// Operands stay as (re, im) pairs: P += a . b and Q += a . swap(b)
// (elementwise, packed FP32x2) hold the four real sums, re phi = P.x - P.y, im
// phi = Q.x + Q.y, so that a product costs two packed FMAs and only b is
// swapped.  Every four pairs of sites (8 terms) groups of eight lanes of a warp
// add their sums up over three levels of a reduce-scatter of shuffles and each
// lane takes eight of the 50 into FP64, where the last two levels follow at the
// end: eight conversions where a lane's own sums would take 50.  A level of the
// tree rounds every sum once, at its whole size where the terms are of one sign
// (orbitals without nodes).  Short sums and three levels keep the error against 64
// bits at or below that of the general kernel, whose chains are 15 terms at n =
// 10, for orbitals of random sign and for positive ones alike; six pairs and five
// levels had 1.8 times its error on positive orbitals (n = 10, L = 24).
//
// What bounds it: at L = 48, n = 10, 128 configurations one read of the
// orbitals takes 173 us and the FMAs 137; measured 440 us (the general kernel,
// 2 x 2 blocks a thread through shared memory: 1012; six pairs and five levels
// 400).  About ten warps per SM (168 registers) wait in turn for a tile's copies,
// the barrier and their own FMAs.  Tiles of 64 sites in six stages: 507 us.
#include <cooperative_groups.h>

#include "lane_sums.cuh"

namespace nrcps {
namespace cg = cooperative_groups;

namespace {

constexpr int SB = 5;           // rows of a block
constexpr int ST = 128;         // sites of a tile
constexpr int SUNITS = ST / 32;
constexpr int SSTAGES = 3;
constexpr int SFLUSH = 4;       // pairs of sites of one FP32 sum
constexpr int SLEVELS = 3;      // levels of the lanes' tree in FP32
constexpr int SWINDOW = 256;    // tiles whose bits are looked up at a time

// NB blocks of rows: warps [0, NB) own the diagonal, the others the blocks
// above it, with NB = 2 two warps (halves of a tile) for the one: 60 products
// per four units against 50.
template <int NB>
struct SymShape {
  static constexpr int ROWS = SB * NB;
  static constexpr int GROUPS = NB == 2 ? 2 : 1;
  static constexpr int OFF = NB * (NB - 1) / 2;
  static constexpr int WARPS = NB + OFF * GROUPS;
  static constexpr int THREADS = 32 * WARPS;
  static constexpr int CTAS = NB == 2 ? 3 : NB == 3 ? 2 : 1;
  static constexpr size_t STAGE = sizeof(float2) * 2 * ROWS * ST + sizeof(float) * ST;
  static constexpr size_t SMEM = SSTAGES * STAGE + sizeof(uint32_t) * (SWINDOW / 32);
  static_assert(sizeof(double) * 64 * WARPS <= SSTAGES * STAGE, "the final sums lie over the stages");
};

__device__ __forceinline__ void copy8(void* dst, const void* src, bool take) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src),
               "r"(take ? 8 : 0)
               : "memory");
}

// A warp's block: all 25 entries, or the 15 of the triangle (DIAG).
struct SymAcc {
  float2 P[SB * SB], Q[SB * SB];
  double sum[64 >> SLEVELS];
  int count;
  template <bool DIAG>
  static __host__ __device__ constexpr int entries() {
    return DIAG ? SB * (SB + 1) / 2 : SB * SB;
  }
  template <bool DIAG>
  static __device__ __forceinline__ constexpr int at(int s, int t) {
    return DIAG ? s * SB - s * (s - 1) / 2 + t - s : s * SB + t;
  }
  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int e = 0; e < SB * SB; ++e) P[e] = Q[e] = make_float2(0.f, 0.f);
    count = 0;
  }
  // w a_s b_t for the block
  template <bool DIAG>
  __device__ __forceinline__ void add(const float2 (&a)[SB], const float2 (&b)[SB], float w) {
    float2 c[SB];
#pragma unroll
    for (int t = 0; t < SB; ++t) c[t] = make_float2(b[t].y, b[t].x);
#pragma unroll
    for (int s = 0; s < SB; ++s) {
      const float2 as = __fmul2_rn(a[s], make_float2(w, w));
#pragma unroll
      for (int t = DIAG ? s : 0; t < SB; ++t) {
        P[at<DIAG>(s, t)] = __ffma2_rn(as, b[t], P[at<DIAG>(s, t)]);
        Q[at<DIAG>(s, t)] = __ffma2_rn(as, c[t], Q[at<DIAG>(s, t)]);
      }
    }
  }
  template <bool DIAG>
  __device__ __forceinline__ void flush(int lane) {
    float v[2 * entries<DIAG>()];
#pragma unroll
    for (int e = 0; e < entries<DIAG>(); ++e) {
      v[2 * e] = P[e].x - P[e].y;
      v[2 * e + 1] = Q[e].x + Q[e].y;
    }
    reduce_scatter<2 * entries<DIAG>(), 0, SLEVELS>(v, lane);
#pragma unroll
    for (int k = 0; k < 32 * lane_share(2 * entries<DIAG>()) >> SLEVELS; ++k) sum[k] += (double)v[k];
    clear();
  }
  // the lanes' FP64 sums over the levels that are left
  template <bool DIAG>
  __device__ __forceinline__ void finish(int lane) {
    flush<DIAG>(lane);
    reduce_scatter<2 * entries<DIAG>(), SLEVELS, 5>(sum, lane);
  }
};

template <int NB>
__global__ void __launch_bounds__(SymShape<NB>::THREADS, SymShape<NB>::CTAS)
    pair_sym_kernel(const float2* __restrict__ psi, int n, long vol, const double* __restrict__ w,
                    const int* __restrict__ opp, const int* __restrict__ flags, double* __restrict__ phi) {
  using Sh = SymShape<NB>;
  if (flags && *flags) return;  // no involution or no even weight: the general kernel's
  extern __shared__ __align__(16) unsigned char ssm[];
  uint32_t* live = reinterpret_cast<uint32_t*>(ssm + SSTAGES * Sh::STAGE);
  cg::cluster_group cluster = cg::this_cluster();
  const int split = (int)cluster.num_blocks(), rank = (int)cluster.block_rank();
  const long conf = blockIdx.x / split;
  const float2* base = psi + (size_t)conf * n * vol;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const long ntiles = (vol + ST - 1) / ST;
  const long mine = ntiles > rank ? (ntiles - rank + split - 1) / split : 0;  // tiles rank, rank + split, ..
  auto stage_x = [&](int b) { return reinterpret_cast<float2*>(ssm + b * Sh::STAGE); };
  // rows past n stay zero
  for (int e = threadIdx.x; e < SSTAGES * (Sh::ROWS - n) * ST; e += Sh::THREADS) {
    float2* x = stage_x(e / ((Sh::ROWS - n) * ST)) + n * ST + e % ((Sh::ROWS - n) * ST);
    x[0] = x[Sh::ROWS * ST] = make_float2(0.f, 0.f);
  }
  // the block of this warp and its share of a tile's units
  const bool diag = warp < NB;
  int bi = warp, bj = warp, unit0 = 0;
  if (!diag) {
    int p = (warp - NB) / Sh::GROUPS;
    unit0 = (warp - NB) % Sh::GROUPS;
    bi = 0;
    while (p >= NB - 1 - bi) {
      p -= NB - 1 - bi;
      ++bi;
    }
    bj = bi + 1 + p;
  }
  SymAcc acc;
  acc.clear();
  for (double& v : acc.sum) v = 0.0;
  for (long win = 0; win < mine; win += SWINDOW) {
    const int tiles = (int)(mine - win < SWINDOW ? mine - win : SWINDOW);
    __syncthreads();
    if (threadIdx.x < SWINDOW / 32) live[threadIdx.x] = 0;
    __syncthreads();
    for (int k = warp; k < tiles; k += Sh::WARPS) {
      const long i0 = (rank + (win + k) * split) * ST;
      bool any = false;
#pragma unroll
      for (int u = 0; u < SUNITS; ++u) {
        const long i = i0 + 32 * u + lane;
        if (i < vol) any |= i <= (long)__ldg(opp + i);
      }
      if (__any_sync(0xffffffffu, any) && lane == 0) atomicOr(live + (k >> 5), 1u << (k & 31));
    }
    __syncthreads();
    // the live tiles in order: `at` walks the bits
    int at = 0;
    auto next = [&]() -> long {
      while (at < tiles) {
        const uint32_t m = live[at >> 5] >> (at & 31);
        if (m) {
          at += __ffs(m);
          return rank + (win + at - 1) * split;
        }
        at = (at & ~31) + 32;
      }
      return -1;
    };
    // partners (and, for the first warps, the weight) of a tile's sites one
    // tile ahead of its copies
    int j[SUNITS];
    float wv = 0.f;
    long tile = next();
    auto look = [&]() {
      if (tile < 0) return;
#pragma unroll
      for (int u = 0; u < SUNITS; ++u) {
        const long i = tile * ST + 32 * u + lane;
        j[u] = i < vol ? __ldg(opp + i) : -1;
      }
      for (int u = warp; u < SUNITS; u += Sh::WARPS) {  // (one unit per warp: WARPS >= SUNITS)
        const long i = tile * ST + 32 * u + lane;
        wv = i < vol ? (float)__ldg(w + i) : 0.f;
      }
    };
    auto issue = [&](int b) {
      if (tile >= 0) {
        float2* x = stage_x(b);
        float* wt = reinterpret_cast<float*>(x + 2 * Sh::ROWS * ST);
        const long i0 = tile * ST + lane;
#pragma unroll
        for (int u = 0; u < SUNITS; ++u) {
          const long i = i0 + 32 * u;
          if (warp == u) wt[32 * u + lane] = i < j[u] ? wv : i == j[u] ? 0.5f * wv : 0.f;
        }
        for (int r = Sh::WARPS - 1 - warp; r < n; r += Sh::WARPS) {  // (the diagonal's warps have the most to sum)
          const float2* row = base + (size_t)r * vol;
#pragma unroll
          for (int u = 0; u < SUNITS; ++u) {
            const long i = i0 + 32 * u;
            const bool take = i <= (long)j[u];
            copy8(x + r * ST + 32 * u + lane, row + (take ? i : 0), take);
            copy8(x + (Sh::ROWS + r) * ST + 32 * u + lane, row + (take ? j[u] : 0), take);
          }
        }
        tile = next();
        look();
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
    };
    int left = 0;  // live tiles of the window
    for (int k = 0; k < SWINDOW / 32; ++k) left += __popc(live[k]);
    look();
#pragma unroll
    for (int b = 0; b < SSTAGES - 1; ++b) issue(b);
    int buf = 0;
    for (; left > 0; --left) {
      asm volatile("cp.async.wait_group %0;" ::"n"(SSTAGES - 2) : "memory");
      __syncthreads();  // this tile is in, and every warp has left the one whose buffer comes next
      issue(buf == 0 ? SSTAGES - 1 : buf - 1);
      const float2* x = stage_x(buf);
      const float2* y = x + Sh::ROWS * ST;
      const float* wt = reinterpret_cast<const float*>(x + 2 * Sh::ROWS * ST);
      if (diag) {
#pragma unroll 1
        for (int u = 0; u < SUNITS; ++u) {
          const int q = 32 * u + lane;
          float2 a[SB], b[SB];
#pragma unroll
          for (int s = 0; s < SB; ++s) {
            a[s] = x[(bi * SB + s) * ST + q];
            b[s] = y[(bi * SB + s) * ST + q];
          }
          acc.add<true>(a, b, wt[q]);
          acc.add<true>(b, a, wt[q]);
          if (++acc.count == SFLUSH) acc.flush<true>(lane);
        }
      } else {
#pragma unroll 1
        for (int u = unit0; u < SUNITS; u += Sh::GROUPS) {
          const int q = 32 * u + lane;
          float2 a[SB], b[SB];
#pragma unroll
          for (int s = 0; s < SB; ++s) {
            a[s] = x[(bi * SB + s) * ST + q];
            b[s] = y[(bj * SB + s) * ST + q];
          }
          acc.add<false>(a, b, wt[q]);
#pragma unroll
          for (int s = 0; s < SB; ++s) {
            a[s] = y[(bi * SB + s) * ST + q];
            b[s] = x[(bj * SB + s) * ST + q];
          }
          acc.add<false>(a, b, wt[q]);
          if (++acc.count == SFLUSH) acc.flush<false>(lane);
        }
      }
      buf = buf == SSTAGES - 1 ? 0 : buf + 1;
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
  }
  if (diag) acc.finish<true>(lane);
  else acc.finish<false>(lane);
  __syncthreads();
  // every warp's sums over the stages, then the cluster's CTAs in rank order
  double* red = reinterpret_cast<double*>(ssm);  // [WARPS][64]
  const int share = lane_share(2 * (diag ? SymAcc::entries<true>() : SymAcc::entries<false>()));
  for (int k = 0; k < share; ++k) red[warp * 64 + share * lane + k] = acc.sum[k];
  cluster.sync();
  for (int e = rank * Sh::THREADS + threadIdx.x; e < 2 * n * n; e += split * Sh::THREADS) {
    const int s = e / 2 / n, t = e / 2 % n, c = e & 1;
    if (s > t) continue;
    const int p = s / SB, q = t / SB;
    double v = 0.0;
    for (int r = 0; r < split; ++r) {
      const double* peer = cluster.map_shared_rank(red, r);
      if (p == q) {
        v += peer[p * 64 + 2 * SymAcc::at<true>(s % SB, t % SB) + c];
      } else {
        const int off = p * (NB - 1) - p * (p - 1) / 2 + (q - p - 1);
        for (int g = 0; g < Sh::GROUPS; ++g)
          v += peer[(NB + off * Sh::GROUPS + g) * 64 + 2 * SymAcc::at<false>(s % SB, t % SB) + c];
      }
    }
    phi[2 * ((conf * n + s) * (long)n + t) + c] = v;
    phi[2 * ((conf * n + t) * (long)n + s) + c] = v;
  }
  cluster.sync();  // peers keep their shared memory until every sum is read
}

// Clusters of `split` CTAs of a kernel that the device runs at a time, asked of the
// driver once per context (its occupancy query takes a few microseconds).
nrcps_status clusters_that_fit(nrcps_context* ctx, const void* kern, int split, int threads, size_t smem, int per_sm,
                               int* fit) {
  int& known = ctx->clusters[{kern, split}];
  if (known) {
    *fit = known;
    return NRCPS_OK;
  }
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)split;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.gridDim = dim3((unsigned)(split * ctx->sm_count));
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (cudaOccupancyMaxActiveClusters(fit, kern, &cfg) != cudaSuccess || *fit < 1) {
    cudaGetLastError();
    *fit = ctx->sm_count * per_sm / split;
    if (*fit < 1) *fit = 1;
  }
  known = *fit;
  return NRCPS_OK;
}

template <int NB>
nrcps_status launch_pair_sym(nrcps_context* ctx, const void* psi, int n, int nconf, long vol, const double* w,
                             const int* opp, const int* flags, double* phi) {
  using Sh = SymShape<NB>;
  auto kern = pair_sym_kernel<NB>;
  NRCPS_TRY(allow_smem(ctx, (const void*)kern, Sh::SMEM, "pair_sym: smem attribute"));
  // the split of a configuration that leaves the fewest rounds of clusters per
  // share, of as many clusters as fit the device (fewer than its SMs divided by
  // the split: a GPC's SMs do not divide by every split)
  const long ntiles = (vol + ST - 1) / ST;
  int split = 1;
  double best = 1e300;
  for (int s = 1; s <= 8 && s <= ntiles; ++s) {
    int fit = 0;
    NRCPS_TRY(clusters_that_fit(ctx, (const void*)kern, s, Sh::THREADS, Sh::SMEM, Sh::CTAS, &fit));
    const double cost = (double)((nconf + fit - 1) / fit) / s;
    if (cost < 0.97 * best) best = cost, split = s;
  }
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)split;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.gridDim = dim3((unsigned)((long)nconf * split));
  cfg.blockDim = dim3(Sh::THREADS);
  cfg.dynamicSmemBytes = Sh::SMEM;
  cfg.stream = ctx->stream;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  ctx->launches++;
  return check_cuda(ctx, cudaLaunchKernelEx(&cfg, kern, reinterpret_cast<const float2*>(psi), n, vol, w, opp, flags,
                                            phi),
                    "pair_sym_kernel launch");
}

}  // namespace

// Below n = 9 the general kernel's chains are short (10 terms at n = 8) and its
// error less than this kernel's; at 11 and 12 also, and three blocks of five rows are
// a quarter padding there.  Below 16^3 sites (n = 16, a fifth padding: 8192) the
// general kernel is the faster one: L = 8, n = 16, 1500 configurations 103 against 211
// us, L = 12, n = 19, 24 of them 23 against 30; from there on this one: L = 16, n = 9,
// one configuration 19 / 19, n = 19, 200 of them 175 against 111, L = 32, n = 10, 64
// 126 against 80.
bool pair_sym_supported(int n, long vol) {
  return n >= 9 && n <= 20 && n != 11 && n != 12 && vol >= (n == 16 ? 8192 : 4096);
}

// flags: the device's check of the table (nonzero: the kernel writes
// nothing), or null where the caller knows that the table qualifies.
nrcps_status pair_sym(nrcps_context* ctx, const void* psi, int n, int nconf, long vol, const double* w, const int* opp,
                      const int* flags, double* phi) {
  return n <= 10   ? launch_pair_sym<2>(ctx, psi, n, nconf, vol, w, opp, flags, phi)
         : n <= 15 ? launch_pair_sym<3>(ctx, psi, n, nconf, vol, w, opp, flags, phi)
                   : launch_pair_sym<4>(ctx, psi, n, nconf, vol, w, opp, flags, phi);
}

}  // namespace nrcps

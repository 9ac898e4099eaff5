// qr.cu -- periodic re-orthonormalisation of the orbitals (CholeskyQR in FP64).
//
// The reference propagates unstabilised (its only option is a host-side
// norm rescale, Propagator::Normalize, src/alg/propagator.C:78-135).  At
// long Euclidean times the orbitals of a configuration align and the Slater
// matrices lose precision.  Here, every qr_period slices, each
// configuration's orbital block Psi (V x N) is replaced by Q with Psi = Q R:
//   G = Psi^H Psi (FP64 accumulation), G = R^H R (Cholesky), Psi <- Psi R^-1.
// R is upper triangular in orbital order, so the first n columns of Psi are
// the first n columns of Q times the leading n x n block of R, and every
// leading-minor determinant the measurement needs is recovered as
//   det S_n(Psi) = det S_n(Q) * prod_{i <= n} R_ii.
// The running sum of log R_ii per orbital is kept per configuration and the
// measured determinants are rescaled by exp(sum_{i<=n} log R_ii).
#include <cooperative_groups.h>

#include "common.cuh"

namespace nrcps {

bool gram_tc_supported(int N, long vol, int nconf);
nrcps_status gram_tc(nrcps_context* ctx, const void* psi, int N, long vol, int nconf, double* G);

// FP64 orbitals: G[c][i][j] for i <= j (the upper triangle the Cholesky reads), one
// block per configuration reading its orbitals once: tiles of GT sites of all N
// orbitals go through shared memory (rows padded by one element so that the
// rows a warp reads fall in different banks); each thread accumulates 2 x 2
// blocks (i, i+1) x (j, j+1) of G over a quarter of each tile's sites, a tile's
// sums apart; the four quarters are summed at the end.
constexpr int GT = 128;
__device__ __forceinline__ void cp_async_elem(cplx<double>* dst, const cplx<double>* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}

// DB: double-buffered tiles (the next tile's asynchronous copies overlap the
// current tile's products); else one tile buffer.
template <int MAXB, bool DB>
__global__ void __launch_bounds__(256) gram_tile_kernel(const void* __restrict__ psi, int N, long vol,
                                                        double* __restrict__ G) {
  typedef cplx<double> cd;
  extern __shared__ __align__(16) unsigned char gsm[];
  cd* tiles = reinterpret_cast<cd*>(gsm);  // [DB ? 2 : 1][N][GT + 1]
  const long c = blockIdx.x;
  const cd* base = reinterpret_cast<const cd*>(psi) + (size_t)c * N * vol;
  const int nb = (N + 1) / 2;                // 2-row blocks
  const int nblk = nb * (nb + 1) / 2;        // upper-triangular block pairs
  const int lane64 = threadIdx.x & 63, grp = threadIdx.x >> 6;
  // MAXB: 2-row block pairs per thread, ceil(nblk / 64): 2 for N <= 22, 3 for N <= 32, 9 for N <= 64
  double acc[MAXB][8];
#pragma unroll
  for (int b = 0; b < MAXB; ++b)
#pragma unroll
    for (int k = 0; k < 8; ++k) acc[b][k] = 0.0;
  auto fill = [&](long p0, cd* t) {
    const int ts = (int)((vol - p0) < GT ? (vol - p0) : GT);
    for (int e = threadIdx.x; e < N * GT; e += blockDim.x) {
      const int i = e / GT, s = e - i * GT;
      if (!DB || s >= ts) t[i * (GT + 1) + s] = s < ts ? base[(size_t)i * vol + p0 + s] : cd{0.0, 0.0};
      else cp_async_elem(t + i * (GT + 1) + s, base + (size_t)i * vol + p0 + s);
    }
    if (DB) asm volatile("cp.async.commit_group;" ::: "memory");
  };
  const size_t tsz = (size_t)N * (GT + 1);
  if (DB) fill(0, tiles);
  int buf = 0;
  for (long p0 = 0; p0 < vol; p0 += GT, buf ^= 1) {
    cd* tile = tiles + (DB ? buf : 0) * tsz;
    if (DB) {
      __syncthreads();  // every thread is done with the tile the next copies overwrite
      if (p0 + GT < vol) fill(p0 + GT, tiles + (buf ^ 1) * tsz);
      else asm volatile("cp.async.commit_group;" ::: "memory");
      asm volatile("cp.async.wait_group 1;" ::: "memory");  // every group but the newest has landed
      __syncthreads();
    } else {
      __syncthreads();
      fill(p0, tile);
      __syncthreads();
    }
#pragma unroll
    for (int b = 0; b < MAXB; ++b) {
      const int blk = lane64 + 64 * b;
      if (blk >= nblk) break;
      // blk -> (bi, bj), bi <= bj, row-major over the upper triangle
      int bi = 0, rem = blk;
      while (rem >= nb - bi) {
        rem -= nb - bi;
        ++bi;
      }
      const int bj = bi + rem;
      const int i0 = 2 * bi, j0 = 2 * bj;
      const int i1 = i0 + 1 < N ? i0 + 1 : i0, j1 = j0 + 1 < N ? j0 + 1 : j0;
      double s[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) s[k] = 0.0;
      for (int q = grp; q < GT; q += 4) {
        const cd a0 = tile[i0 * (GT + 1) + q], a1 = tile[i1 * (GT + 1) + q];
        const cd b0 = tile[j0 * (GT + 1) + q], b1 = tile[j1 * (GT + 1) + q];
        // conj(a) b: two fused multiply-adds per component
        s[0] = fma(a0.re, b0.re, s[0]);
        s[0] = fma(a0.im, b0.im, s[0]);
        s[1] = fma(a0.re, b0.im, s[1]);
        s[1] = fma(-a0.im, b0.re, s[1]);
        s[2] = fma(a0.re, b1.re, s[2]);
        s[2] = fma(a0.im, b1.im, s[2]);
        s[3] = fma(a0.re, b1.im, s[3]);
        s[3] = fma(-a0.im, b1.re, s[3]);
        s[4] = fma(a1.re, b0.re, s[4]);
        s[4] = fma(a1.im, b0.im, s[4]);
        s[5] = fma(a1.re, b0.im, s[5]);
        s[5] = fma(-a1.im, b0.re, s[5]);
        s[6] = fma(a1.re, b1.re, s[6]);
        s[6] = fma(a1.im, b1.im, s[6]);
        s[7] = fma(a1.re, b1.im, s[7]);
        s[7] = fma(-a1.im, b1.re, s[7]);
      }
#pragma unroll
      for (int k = 0; k < 8; ++k) acc[b][k] += s[k];
    }
  }
  // sum the four site quarters through shared memory, write the upper triangle
  __syncthreads();
  double* red = reinterpret_cast<double*>(gsm);  // [nblk][8] (fits: tile area >= 9 KB)
  for (int g = 0; g < 4; ++g) {
    if (grp == g) {
#pragma unroll
      for (int b = 0; b < MAXB; ++b) {
        const int blk = lane64 + 64 * b;
        if (blk >= nblk) break;
#pragma unroll
        for (int k = 0; k < 8; ++k) red[blk * 8 + k] = (g == 0 ? 0.0 : red[blk * 8 + k]) + acc[b][k];
      }
    }
    __syncthreads();
  }
  for (int blk = threadIdx.x; blk < nblk; blk += blockDim.x) {
    int bi = 0, rem = blk;
    while (rem >= nb - bi) {
      rem -= nb - bi;
      ++bi;
    }
    const int bj = bi + rem;
    for (int u = 0; u < 2; ++u)
      for (int v = 0; v < 2; ++v) {
        const int i = 2 * bi + u, j = 2 * bj + v;
        if (i >= N || j >= N || i > j) continue;
        double* g = G + 2 * ((c * N + i) * (long)N + j);
        g[0] = red[blk * 8 + 4 * u + 2 * v];
        g[1] = red[blk * 8 + 4 * u + 2 * v + 1];
      }
  }
}

// Per configuration: Cholesky G = R^H R (R upper), Rinv = R^{-1}, and
// logR[c][i] += log R_ii; G is overwritten with Rinv.  A non-positive pivot
// marks the configuration with NaN in logR (and leaves its G as far as it
// got).  f32_apply: the orbitals are FP32 and Rinv will be applied rounded to
// FP32; the leading-minor identity det S_n(Psi) = det S_n(Psi Rinv) /
// prod_{i<n} Rinv_ii then holds for the ROUNDED diagonal, so logR accumulates
// -log(float(Rinv_ii)) instead of log R_ii.
//
// One block per configuration, the matrix in shared memory: the columns below
// a pivot are updated by all threads at once, every entry in the order of the
// sum over k (right-looking; the values a left-looking factorisation has), and
// each row of the inverse by one thread per column.  A serial chain of N
// square roots and divisions is left: 29 us for 256 matrices of N = 19, 34 us
// for 1024 (one thread per matrix: 610 and 675 us).
constexpr int CHOL_THREADS = 128;  // a warp for N <= 8
__global__ void __launch_bounds__(CHOL_THREADS) chol_inv_kernel(double* __restrict__ G, int N,
                                                                double* __restrict__ logR, int f32_apply) {
  extern __shared__ double2 cm[];  // [N][N]
  const long c = blockIdx.x;
  const int threads = (int)blockDim.x;
  double* g = G + 2 * c * N * N;  // (the caller's work buffer: doubles, not on 16 bytes of need)
  auto write_back = [&]() {
    for (int e = threadIdx.x; e < N * N; e += threads)
      if (e / N <= e % N) {
        g[2 * e] = cm[e].x;
        g[2 * e + 1] = cm[e].y;
      }
  };
  for (int e = threadIdx.x; e < N * N; e += threads)
    if (e / N <= e % N) cm[e] = make_double2(g[2 * e], g[2 * e + 1]);
  __syncthreads();
  bool ok = true;
  for (int k = 0; k < N; ++k) {
    const double d = cm[k * N + k].x;
    if (!(d > 0.0)) {  // (the same for every thread)
      ok = false;
      break;
    }
    const double rkk = sqrt(d);
    __syncthreads();  // every thread has read the pivot
    for (int j = k + threadIdx.x; j < N; j += threads) {
      if (j == k) cm[k * N + k] = make_double2(rkk, 0.0);
      else cm[k * N + j] = make_double2(cm[k * N + j].x / rkk, cm[k * N + j].y / rkk);
    }
    __syncthreads();
    // G_ij -= conj(R_ki) R_kj for k < i <= j
    const int m = N - k - 1;
    for (int e = threadIdx.x; e < m * m; e += threads) {
      const int i = k + 1 + e / m, j = k + 1 + e % m;
      if (i > j) continue;
      const double2 a = cm[k * N + i], b = cm[k * N + j];
      double2 v = cm[i * N + j];
      if (i == j) {
        v.x -= a.x * a.x + a.y * a.y;
      } else {
        v.x -= a.x * b.x + a.y * b.y;
        v.y -= a.x * b.y - a.y * b.x;
      }
      cm[i * N + j] = v;
    }
    __syncthreads();
  }
  if (!ok) {
    write_back();
    for (int i = threadIdx.x; i < N; i += threads) logR[c * N + i] = nan("");
    return;
  }
  if (!f32_apply)
    for (int i = threadIdx.x; i < N; i += threads) logR[c * N + i] += log(cm[i * N + i].x);
  __syncthreads();
  // Rinv in place, row by row from the bottom: Rinv_ii = 1 / R_ii,
  // Rinv_ij = -(sum_{k=i+1..j} R_ik Rinv_kj) / R_ii for j > i (a thread per j;
  // N is at most the threads)
  for (int i = N - 1; i >= 0; --i) {
    const double rii = cm[i * N + i].x;
    const int j = i + 1 + threadIdx.x;
    double sr = 0, si = 0;
    if (j < N)
      for (int k = i + 1; k <= j; ++k) {
        const double2 a = cm[i * N + k], b = cm[k * N + j];
        sr += a.x * b.x - a.y * b.y;
        si += a.x * b.y + a.y * b.x;
      }
    __syncthreads();  // row i has been read
    if (j < N) cm[i * N + j] = make_double2(-sr / rii, -si / rii);
    if (threadIdx.x == 0) cm[i * N + i] = make_double2(1.0 / rii, 0.0);
    __syncthreads();
  }
  if (f32_apply)
    for (int i = threadIdx.x; i < N; i += threads) logR[c * N + i] -= log((double)(float)cm[i * N + i].x);
  write_back();
}

// FP32 orbitals.  One cluster of CTAs per configuration (and group of 16 block
// pairs), each CTA a share of the sites; thread (slot, l) accumulates one
// 4 x 4 block (rows 4 bi.., columns 4 bj.., bi <= bj) of G.  A stage of sites
// goes from HBM through registers (the next stage's loads are in flight during
// this one's products) into shared memory with real and imaginary parts apart,
// so that a packed FP32x2 operand is the same part of two neighbouring sites:
// 16 eight-byte loads feed 64 packed FMAs and no register is copied into a
// pair.  Every FP32 sum runs over 32 sites, then goes into FP64 sums, which
// wait in shared memory (32 per thread: in registers they would take the
// place of the FP32 block).  Lanes, groups and CTAs are summed in a fixed
// order; the split depends on the volume alone, so a configuration's G does
// not depend on the batch it is in.
// Bounds at N = 19, L = 32, 1024 configurations: one read of the orbitals 0.78
// ms, the FMA pipe 1.2 ms (960 FMAs per site), the shared-memory loads about
// the same.  Measured 2.61 ms (FMA pipe 45 %: the loads of a block and its
// FMAs overlap in part only at 16 warps per SM); 3.07 ms with the (re, im)
// pair of one site as the packed operand, which copies registers into pairs.
// The split over a cluster serves small batches: 256 configurations 0.70 ms
// against 0.90 (one CTA per configuration leaves 40 SMs half empty), N = 24,
// 64 configurations at L = 24, whole call: 0.27 against 1.84.
constexpr int G4_THREADS = 256;
constexpr int G4_LANES = 16;                       // site lanes per slot
constexpr int G4_SLOTS = G4_THREADS / G4_LANES;    // block pairs in flight
constexpr int G4_FLUSH = 32;                       // sites per FP32 sum
// sites per stage: small N leave slots free, which then share the stage's
// sites (G groups per block pair)
constexpr int g4_sites(int nb) { return nb == 1 ? 512 : nb <= 5 ? 128 : 64; }
constexpr int g4_groups(int nb) { return nb == 1 ? 16 : nb == 2 ? 4 : nb == 3 ? 2 : 1; }
constexpr int g4_chunks(int nb) { return (4 * nb * g4_sites(nb) / 2 + G4_THREADS - 1) / G4_THREADS; }
constexpr size_t g4_smem(int nb) {
  return sizeof(float) * 2 * 2 * 4 * nb * g4_sites(nb) + sizeof(double) * 32 * G4_THREADS;
}

template <int nb>  // blocks of four rows
__global__ void __launch_bounds__(G4_THREADS, 2) gram4_kernel(const float2* __restrict__ psi, int N, long vol,
                                                              int aligned, double* __restrict__ G) {
  extern __shared__ __align__(16) unsigned char gsm[];
  namespace cg = cooperative_groups;
  cg::cluster_group cluster = cg::this_cluster();
  const int split = (int)cluster.num_blocks(), rank = (int)cluster.block_rank();
  const long c = blockIdx.x / split;
  constexpr int npairs = nb * (nb + 1) / 2, rows = 4 * nb, T = g4_sites(nb), groups = g4_groups(nb);
  constexpr int NCH = g4_chunks(nb);  // two-site pieces of a stage per thread
  double* acc = reinterpret_cast<double*>(gsm);  // [32][G4_THREADS]
  float* tiles = reinterpret_cast<float*>(acc + 32 * G4_THREADS);  // [2][re, im][rows][T]
  constexpr int plane = rows * T, halfT = T / 2;
  const float2* base = psi + (size_t)c * N * vol;
  const int l = threadIdx.x % G4_LANES, slot = threadIdx.x / G4_LANES;
  const int first = (int)blockIdx.y * G4_SLOTS;
  const int here = npairs - first < G4_SLOTS ? npairs - first : G4_SLOTS;  // pairs of this CTA
  const int grp = slot / here;
  const bool active = grp < groups;
  int bi = 0, rem = active ? first + slot % here : 0;
  while (rem >= nb - bi) {
    rem -= nb - bi;
    ++bi;
  }
  const int bj = bi + rem;
#pragma unroll
  for (int k = 0; k < 32; ++k) acc[k * G4_THREADS + threadIdx.x] = 0.0;
  // this CTA's stages
  const long stages = (vol + T - 1) / T;
  const long s0 = stages * rank / split, s1 = stages * (rank + 1) / split;
  // piece e of a stage: sites 2 j, 2 j + 1 of row i
  float4 pre[NCH];
  auto load = [&](long st) {
#pragma unroll
    for (int u = 0; u < NCH; ++u) {
      const int e = threadIdx.x + u * G4_THREADS, i = e / halfT;
      const long p = st * T + 2 * (e - i * halfT);
      pre[u] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (i < N) {
        const float2* q = base + (size_t)i * vol + p;
        if (aligned && p + 1 < vol) {
          pre[u] = __ldcs(reinterpret_cast<const float4*>(q));
        } else {
          if (p < vol) pre[u].x = q[0].x, pre[u].y = q[0].y;
          if (p + 1 < vol) pre[u].z = q[1].x, pre[u].w = q[1].y;
        }
      }
    }
  };
  auto store = [&](float* t) {
#pragma unroll
    for (int u = 0; u < NCH; ++u) {
      const int e = threadIdx.x + u * G4_THREADS;
      if (e < rows * halfT) {
        reinterpret_cast<float2*>(t)[e] = make_float2(pre[u].x, pre[u].z);
        reinterpret_cast<float2*>(t + plane)[e] = make_float2(pre[u].y, pre[u].w);
      }
    }
  };
  float2 sr[16], si[16];
#pragma unroll
  for (int k = 0; k < 16; ++k) sr[k] = si[k] = make_float2(0.f, 0.f);
  int summed = 0;
  auto flush = [&]() {
#pragma unroll
    for (int k = 0; k < 16; ++k) {
      double* d = acc + 2 * k * G4_THREADS + threadIdx.x;
      d[0] += (double)sr[k].x + (double)sr[k].y;
      d[G4_THREADS] += (double)si[k].x + (double)si[k].y;
      sr[k] = si[k] = make_float2(0.f, 0.f);
    }
    summed = 0;
  };
  if (s0 < s1) load(s0);
  int buf = 0;
  for (long st = s0; st < s1; ++st, buf ^= 1) {
    float* t = tiles + buf * 2 * plane;
    store(t);
    if (st + 1 < s1) load(st + 1);
    // (a thread stores into this buffer again only after the next stage's
    // barrier, which every reader of this stage has then reached)
    __syncthreads();
    if (active) {
      for (int ch = grp; ch < T / 32; ch += groups) {
        const float* ta = t + 4 * bi * T + 32 * ch + 2 * l;
        const float* tb = t + 4 * bj * T + 32 * ch + 2 * l;
        float2 br[4], bm[4];
#pragma unroll
        for (int v = 0; v < 4; ++v) {
          br[v] = *reinterpret_cast<const float2*>(tb + v * T);
          bm[v] = *reinterpret_cast<const float2*>(tb + plane + v * T);
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const float2 ar = *reinterpret_cast<const float2*>(ta + u * T);
          const float2 am = *reinterpret_cast<const float2*>(ta + plane + u * T);
          const float2 nm = make_float2(-am.x, -am.y);
          // conj(a) b = (ar br + am bm) + i (ar bm - am br)
#pragma unroll
          for (int v = 0; v < 4; ++v) {
            sr[4 * u + v] = __ffma2_rn(ar, br[v], sr[4 * u + v]);
            si[4 * u + v] = __ffma2_rn(ar, bm[v], si[4 * u + v]);
          }
#pragma unroll
          for (int v = 0; v < 4; ++v) {
            sr[4 * u + v] = __ffma2_rn(am, bm[v], sr[4 * u + v]);
            si[4 * u + v] = __ffma2_rn(nm, br[v], si[4 * u + v]);
          }
        }
        if (++summed == G4_FLUSH) flush();
      }
    }
  }
  flush();
  __syncthreads();
  // the lanes and groups of every pair, then the cluster's CTAs
  double* red = reinterpret_cast<double*>(tiles);  // [here][32], over the stages
  static_assert(groups <= 2 || sizeof(double) * npairs * 32 * (G4_LANES + 1) <= sizeof(float) * 4 * plane, "sums over the stages");
  if (groups > 2) {  // the groups of an entry and lane first, by all threads (256 sums in a row took 3 us)
    double* lanes = red + here * 32;  // [here][32][G4_LANES]
    for (int e = threadIdx.x; e < here * 32 * G4_LANES; e += G4_THREADS) {
      const int j = e % G4_LANES, k = e / G4_LANES % 32, pr = e / G4_LANES / 32;
      double v = 0.0;
      for (int g = 0; g < groups; ++g) v += acc[k * G4_THREADS + (g * here + pr) * G4_LANES + j];
      lanes[e] = v;
    }
    __syncthreads();
  }
  for (int e = threadIdx.x; e < here * 32; e += G4_THREADS) {
    const int pr = e / 32, k = e % 32;
    const double* from = groups > 2 ? red + here * 32 + e * G4_LANES : acc + k * G4_THREADS + pr * G4_LANES;
    double v = 0.0;
    for (int g = 0; g < (groups > 2 ? 1 : groups); ++g)
      for (int j = 0; j < G4_LANES; ++j) v += from[g * here * G4_LANES + j];
    red[e] = v;
  }
  cluster.sync();
  // entries spread over the CTAs
  for (int e = rank * G4_THREADS + threadIdx.x; e < here * 32; e += split * G4_THREADS) {
    double v = 0.0;
    for (int r = 0; r < split; ++r) v += cluster.map_shared_rank(red, r)[e];
    int x = 0, y = first + e / 32;
    while (y >= nb - x) {
      y -= nb - x;
      ++x;
    }
    const int k = (e % 32) / 2, i = 4 * x + k / 4, j = 4 * (x + y) + k % 4;
    if (i < N && j < N && i <= j) G[2 * ((c * N + i) * (long)N + j) + (e & 1)] = v;
  }
  cluster.sync();  // peers keep their shared memory until every sum is read
}

// psi_{c,t}(p) <- sum_{i <= t} psi_{c,i}(p) Rinv[i][t]; one thread per site,
// all N orbitals of a configuration in registers (N <= 64), arithmetic in R
// (FP32 orbitals: Rinv rounded to FP32, see chol_inv_kernel).
template <typename R, int NMAX>
__global__ void __launch_bounds__(256) apply_rinv_kernel(void* __restrict__ psi, int N, long vol, int nconf,
                                                          const double* __restrict__ Rinv) {
  // R^-1 of this block's configuration: 2 N^2 values in R (FP64), or for FP32
  // N^2 float4 (re, re, im, im) entries that feed packed FMAs
  extern __shared__ __align__(16) double rs_raw[];
  R* rs = reinterpret_cast<R*>(rs_raw);
  const long sites_per_block = blockDim.x;
  const long blocks_per_conf = (vol + sites_per_block - 1) / sites_per_block;
  const long c = blockIdx.x / blocks_per_conf;
  if (c >= nconf) return;
  const long p = (blockIdx.x % blocks_per_conf) * sites_per_block + threadIdx.x;
  const bool live = p < vol;
  cplx<R>* base = reinterpret_cast<cplx<R>*>(psi) + (size_t)c * N * vol + (live ? p : 0);
  // the orbital loads go out first; their latency covers the fill of R below
  R xr[NMAX], xi[NMAX];
#pragma unroll
  for (int i = 0; i < NMAX; ++i)
    if (i < N && live) {
      cplx<R> v = base[(size_t)i * vol];
      xr[i] = v.re;
      xi[i] = v.im;
    }
  if constexpr (sizeof(R) == 4) {
    // x r = (xr ar - xi ai, xr ai + xi ar): with X = (xr, xi) the packed sums
    // s = sum X (ar, ar) and u = sum X (ai, ai) give re = s.x - u.y, im = s.y + u.x
    float4* r4 = reinterpret_cast<float4*>(rs_raw);
    for (int e = threadIdx.x; e < N * N; e += blockDim.x) {
      const float ar = (float)Rinv[2L * (c * N * N + e)], ai = (float)Rinv[2L * (c * N * N + e) + 1];
      r4[e] = make_float4(ar, ar, ai, ai);
    }
    __syncthreads();
    if (!live) return;
#pragma unroll
    for (int t = NMAX - 1; t >= 0; --t) {
      if (t >= N) continue;
      float2 sa = make_float2(0.f, 0.f), ua = make_float2(0.f, 0.f);
#pragma unroll
      for (int i = 0; i <= t; ++i) {
        const float4 r = r4[i * N + t];
        const float2 x = make_float2(xr[i], xi[i]);
        sa = __ffma2_rn(x, make_float2(r.x, r.y), sa);
        ua = __ffma2_rn(x, make_float2(r.z, r.w), ua);
      }
      base[(size_t)t * vol] = cplx<R>{sa.x - ua.y, sa.y + ua.x};
    }
  } else {
    for (int e = threadIdx.x; e < 2 * N * N; e += blockDim.x) rs[e] = (R)Rinv[2L * c * N * N + e];
    __syncthreads();
    if (!live) return;
#pragma unroll
    for (int t = NMAX - 1; t >= 0; --t) {
      if (t >= N) continue;
      R sr = 0, si = 0;
#pragma unroll
      for (int i = 0; i <= t; ++i) {
        const R ar = rs[2 * (i * N + t)], ai = rs[2 * (i * N + t) + 1];
        sr = fma(xr[i], ar, sr);
        sr = fma(-xi[i], ai, sr);
        si = fma(xr[i], ai, si);
        si = fma(xi[i], ar, si);
      }
      base[(size_t)t * vol] = cplx<R>{(R)sr, (R)si};
    }
  }
}

// The same for FP32 orbitals and N <= 24, two neighbouring sites per thread:
// 16-byte loads and stores, and each entry of R^-1 read from shared memory
// serves four packed FMAs.  Bound by HBM (one read, one write): 1024
// configurations of N = 19 at L = 32 take 2.15 ms, 4.75 TB/s, 0.73 of a copy
// (one site per thread: 2.27 ms).
template <int NMAX>
__global__ void __launch_bounds__(128) apply_rinv2_kernel(float2* __restrict__ psi, int N, long vol,
                                                          const double* __restrict__ Rinv) {
  __shared__ float4 r4[NMAX * NMAX];  // (re, re, im, im)
  const long blocks_per_conf = (vol / 2 + 127) / 128;
  const long c = blockIdx.x / blocks_per_conf;
  const long p = 2 * ((blockIdx.x % blocks_per_conf) * 128 + threadIdx.x);
  const bool live = p < vol;
  float2* base = psi + (size_t)c * N * vol + (live ? p : 0);
  float4 x[NMAX];
#pragma unroll
  for (int i = 0; i < NMAX; ++i)
    if (i < N && live) x[i] = *reinterpret_cast<const float4*>(base + (size_t)i * vol);
  for (int e = threadIdx.x; e < N * N; e += 128) {
    const float ar = (float)Rinv[2L * (c * N * N + e)], ai = (float)Rinv[2L * (c * N * N + e) + 1];
    r4[e] = make_float4(ar, ar, ai, ai);
  }
  __syncthreads();
  if (!live) return;
#pragma unroll
  for (int t = NMAX - 1; t >= 0; --t) {
    if (t >= N) continue;
    float2 s0 = make_float2(0.f, 0.f), u0 = s0, s1 = s0, u1 = s0;
#pragma unroll
    for (int i = 0; i <= t; ++i) {
      const float4 r = r4[i * N + t];
      const float2 rr = make_float2(r.x, r.y), ri = make_float2(r.z, r.w);
      const float2 x0 = make_float2(x[i].x, x[i].y), x1 = make_float2(x[i].z, x[i].w);
      s0 = __ffma2_rn(x0, rr, s0);
      u0 = __ffma2_rn(x0, ri, u0);
      s1 = __ffma2_rn(x1, rr, s1);
      u1 = __ffma2_rn(x1, ri, u1);
    }
    *reinterpret_cast<float4*>(base + (size_t)t * vol) =
        make_float4(s0.x - u0.y, s0.y + u0.x, s1.x - u1.y, s1.y + u1.x);
  }
}

// The determinants measured at slice t on the re-orthonormalised orbitals
// Q = Psi R^-1, turned into those of Psi, with S_n = sum_{i<=n} log R_ii:
//  mode 0 (SlaterDet::Run, S = <src|Psi> = <src|Q> R):
//    dets[c][t][n]    *= exp(S_n)                      (det S_{n+1})
//  mode 1 (SlaterDet2::Run on the pair matrix Phi(Psi) = R^T Phi(Q) R, whose
//  column n is replaced by v_s = <src_n|psi_s>, v(Psi) = R^T v(Q)):
//    dets[c][t][2n+1] *= exp(2 S_n)                    (det Phi_{n+1})
//    dets[c][t][2n]   *= exp(S_n + S_{n-1})            (det R_{n+1} det R_n)
// (slater_det2.C:78-148; R upper triangular, so the leading blocks of R^T
// Phi R involve only the leading blocks of R).
__global__ void rescale_dets_kernel(double* dets, const double* logR, int N, int nconf, long conf_stride,
                                    long offset, int mode) {
  const long total = (long)nconf * N;
  for (long e = (long)blockIdx.x * blockDim.x + threadIdx.x; e < total; e += (long)gridDim.x * blockDim.x) {
    const long c = e / N;
    const int n = (int)(e % N);
    double s = 0;
    for (int i = 0; i < n; ++i) s += logR[c * N + i];
    const double s_prev = s;  // S_{n-1}
    s += logR[c * N + n];     // S_n
    double* base = dets + c * conf_stride + offset;
    if (mode == 0) {
      const double f = exp(s);
      base[2L * n] *= f;
      base[2L * n + 1] *= f;
    } else {
      const double f1 = exp(2.0 * s), f0 = exp(s + s_prev);
      base[2L * (2 * n + 1)] *= f1;
      base[2L * (2 * n + 1) + 1] *= f1;
      base[2L * (2 * n)] *= f0;
      base[2L * (2 * n) + 1] *= f0;
    }
  }
}

constexpr size_t kMatrixSmem = sizeof(double2) * 64 * 64;  // N <= 64

template <int NMAX>
static nrcps_status launch_apply(nrcps_context* ctx, void* psi, int N, long vol, int nconf, nrcps_precision prec,
                                 const double* Rinv) {
  if constexpr (NMAX <= 24) {
    if (prec == NRCPS_F32 && vol % 2 == 0 && (reinterpret_cast<uintptr_t>(psi) & 15) == 0) {
      apply_rinv2_kernel<NMAX><<<(unsigned)((vol / 2 + 127) / 128 * nconf), 128, 0, ctx->stream>>>(
          reinterpret_cast<float2*>(psi), N, vol, Rinv);
      ctx->launches++;
      return check_launch(ctx, "apply_rinv2_kernel");
    }
  }
  const long bpc = (vol + 255) / 256;
  const size_t sh = sizeof(double) * 2 * N * N;
  if (sh > 48 * 1024) {
    const void* kern = prec == NRCPS_F64 ? (const void*)apply_rinv_kernel<double, NMAX>
                                         : (const void*)apply_rinv_kernel<float, NMAX>;
    NRCPS_TRY(allow_smem(ctx, kern, kMatrixSmem, "apply_rinv_kernel: smem attribute"));
  }
  if (prec == NRCPS_F64)
    apply_rinv_kernel<double, NMAX><<<(unsigned)(bpc * nconf), 256, sh, ctx->stream>>>(psi, N, vol, nconf, Rinv);
  else
    apply_rinv_kernel<float, NMAX><<<(unsigned)(bpc * nconf), 256, sh, ctx->stream>>>(psi, N, vol, nconf, Rinv);
  ctx->launches++;
  return check_launch(ctx, "apply_rinv_kernel");
}

static nrcps_status launch_gram4(nrcps_context* ctx, const void* psi, int N, long vol, int nconf, double* G) {
  const int nb = (N + 3) / 4, npairs = nb * (nb + 1) / 2;
  const size_t sh = g4_smem(nb);
  void (*kern)(const float2*, int, long, int, double*) = nullptr;
  switch (nb) {
#define NRCPS_CASE(B) \
  case B:             \
    kern = gram4_kernel<B>; \
    break;
    NRCPS_CASE(1) NRCPS_CASE(2) NRCPS_CASE(3) NRCPS_CASE(4) NRCPS_CASE(5) NRCPS_CASE(6) NRCPS_CASE(7) NRCPS_CASE(8)
    NRCPS_CASE(9) NRCPS_CASE(10) NRCPS_CASE(11) NRCPS_CASE(12) NRCPS_CASE(13) NRCPS_CASE(14) NRCPS_CASE(15)
    NRCPS_CASE(16)
#undef NRCPS_CASE
  }
  NRCPS_TRY(allow_smem(ctx, (const void*)kern, sh, "gram4: smem attribute"));
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  // CTAs per configuration: at least 16 stages each
  const long stages = vol / g4_sites(nb);
  attr[0].val.clusterDim.x = stages >= 128 ? 8 : stages >= 64 ? 4 : stages >= 32 ? 2 : 1;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.gridDim = dim3((unsigned)nconf * attr[0].val.clusterDim.x, (unsigned)((npairs + G4_SLOTS - 1) / G4_SLOTS));
  cfg.blockDim = dim3(G4_THREADS);
  cfg.dynamicSmemBytes = sh;
  cfg.stream = ctx->stream;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  // 16-byte loads need rows that start on 16 bytes
  const int aligned = (reinterpret_cast<uintptr_t>(psi) & 15) == 0 && vol % 2 == 0;
  return check_cuda(ctx, cudaLaunchKernelEx(&cfg, kern, reinterpret_cast<const float2*>(psi), N, vol, aligned, G),
                    "gram4_kernel");
}

static nrcps_status launch_gram_tile(nrcps_context* ctx, const void* psi, int N, long vol, int nconf, double* G) {
  const size_t tile_bytes = sizeof(cplx<double>) * (size_t)N * (GT + 1);
  const bool db = 2 * tile_bytes <= 200 * 1024;
  size_t sh = db ? 2 * tile_bytes : tile_bytes;
  const size_t red = sizeof(double) * 8 * 528;
  if (sh < red) sh = red;
  auto launch = [&](auto kern) -> nrcps_status {
    NRCPS_TRY(allow_smem(ctx, (const void*)kern, 200 * 1024, "gram_tile_kernel: smem attribute"));
    kern<<<(unsigned)nconf, 256, sh, ctx->stream>>>(psi, N, vol, G);
    return check_launch(ctx, "gram_tile_kernel");
  };
  if (N <= 22) return launch(gram_tile_kernel<2, true>);
  if (N <= 32) return launch(gram_tile_kernel<3, true>);
  return db ? launch(gram_tile_kernel<9, true>) : launch(gram_tile_kernel<9, false>);
}

// One re-orthonormalisation of nconf configurations of N orbitals.
// G: scratch of nconf * N * N complex doubles; logR accumulates.
nrcps_status qr_reorthonormalise(nrcps_context* ctx, void* psi, int N, long vol, int nconf, nrcps_precision prec,
                                 double* G, double* logR) {
  if (N > 64) return set_error(ctx, NRCPS_ERR_UNSUPPORTED, "QR re-orthonormalisation supports N <= 64");
  if (prec == NRCPS_F32 && ctx->qr_gram_tc && gram_tc_supported(N, vol, nconf)) {
    NRCPS_TRY(gram_tc(ctx, psi, N, vol, nconf, G));  // tcgen05, TF32 hi/lo (gram_tc.cu)
  } else {
    NRCPS_TRY(prec == NRCPS_F64 ? launch_gram_tile(ctx, psi, N, vol, nconf, G) : launch_gram4(ctx, psi, N, vol, nconf, G));
    ctx->launches++;
  }
  const size_t chol_sh = sizeof(double2) * N * N;
  if (chol_sh > 48 * 1024)
    NRCPS_TRY(allow_smem(ctx, (const void*)chol_inv_kernel, kMatrixSmem, "chol_inv_kernel: smem attribute"));
  chol_inv_kernel<<<(unsigned)nconf, N <= 8 ? 32 : CHOL_THREADS, chol_sh, ctx->stream>>>(G, N, logR, prec == NRCPS_F32);
  ctx->launches++;
  NRCPS_TRY(check_launch(ctx, "chol_inv_kernel"));
  if (N <= 8) return launch_apply<8>(ctx, psi, N, vol, nconf, prec, G);
  if (N <= 16) return launch_apply<16>(ctx, psi, N, vol, nconf, prec, G);
  if (N <= 24) return launch_apply<24>(ctx, psi, N, vol, nconf, prec, G);
  if (N <= 40) return launch_apply<40>(ctx, psi, N, vol, nconf, prec, G);
  return launch_apply<64>(ctx, psi, N, vol, nconf, prec, G);
}

nrcps_status rescale_dets(nrcps_context* ctx, double* dets, const double* logR, int N, int nconf, long conf_stride,
                          long offset, int mode) {
  rescale_dets_kernel<<<grid_for((long)nconf * N, 256), 256, 0, ctx->stream>>>(dets, logR, N, nconf, conf_stride,
                                                                               offset, mode);
  ctx->launches++;
  return check_launch(ctx, "rescale_dets_kernel");
}

}  // namespace nrcps

using namespace nrcps;

extern "C" nrcps_status nrcps_reorthonormalise(nrcps_context* ctx, void* dev_psi, int N, long vol, int nconf,
                                               nrcps_precision prec, double* dev_work, double* dev_logR) {
  if (!ctx) return NRCPS_ERR_INVALID_ARGUMENT;
  NRCPS_REQUIRE(ctx, N > 0 && vol > 0 && nconf >= 0 && (prec == NRCPS_F32 || prec == NRCPS_F64),
                "nrcps_reorthonormalise: bad arguments");
  if (nconf == 0) return NRCPS_OK;
  NRCPS_REQUIRE(ctx, dev_psi && dev_work && dev_logR, "nrcps_reorthonormalise: null pointer");
  return qr_reorthonormalise(ctx, dev_psi, N, vol, nconf, prec, dev_work, dev_logR);
}

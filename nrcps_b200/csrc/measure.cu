// measure.cu -- Slater-matrix fills and determinants (the measurement half of
// every time slice): overlaps S = <src|psi>, the pair matrix of TwoBody, and
// FP64 LU of every leading minor with the reference's pivoting rule.
#include <cooperative_groups.h>

#include <type_traits>
#include "common.cuh"

namespace nrcps {
namespace cg = cooperative_groups;

// ---------------------------------------------------------------- overlap
// S[c][s][t] = sum_p conj(src_s(p)) psi_{c,t}(p) in FP64 for both orbital
// precisions.  A CTA takes consecutive chunks of one configuration's sites and a
// tile of up to 32 blocks of 4 sources x 4 orbitals; stages of T sites of all its
// rows pass through shared memory (cp.async, two buffers), thread (block, l)
// sums its block over the sites l, l + lanes, ..: 8 sixteen-byte loads for 64
// FP64 FMAs.
//
// The order of every sum is given by (ns, nt, vol) alone, so that a
// configuration's overlap has the same bits in every batch, on every stream and
// in a graph: a chunk by the lanes, then their tree; the chunks of a group (an
// eighth) one after the other; the groups one after the other.  Who does which
// is free: one CTA all of a configuration, a cluster a group per CTA, or, where
// few configurations leave the chip idle, a CTA a few chunks whose sums go to
// `out` one by one and overlap_sum_kernel adds up; or overlap_direct_kernel.
//
// Why chunks: one configuration's overlap is 47 M FP64 FMAs at N = 19, L = 32,
// 3 us of the whole chip, and the reference's drivers measure one
// configuration at a time.  Measured (FP64, call by call): that one 34 us, most
// of it launch and latency (a block per orbital: 216); 40 configurations 0.36
// ms against 1.06, 300 2.51 against 6.89, 30 % of the FP64 pipe, where the
// shared-memory loads (45 %), the barriers of a stage and the FMAs take turns.
constexpr int OV_THREADS = 256;

struct OvTile {
  int ts, tt;        // blocks of a tile along sources and orbitals
  int ns_t, nt_t;    // tiles along each
  int rows, T, lanes;
  int log_t;         // T = 1 << log_t
};
static OvTile overlap_tiles(int ns, int nt) {
  OvTile o;
  const int bs = (ns + 3) / 4, bt = (nt + 3) / 4;
  if (bs * bt <= 32) {
    o.ts = bs, o.tt = bt;
  } else {  // near-equal tiles of at most 5 x 6 blocks
    const int ks = (bs + 4) / 5, kt = (bt + 5) / 6;
    o.ts = (bs + ks - 1) / ks, o.tt = (bt + kt - 1) / kt;
  }
  o.ns_t = (bs + o.ts - 1) / o.ts, o.nt_t = (bt + o.tt - 1) / o.tt;
  o.rows = 4 * (o.ts + o.tt);
  o.lanes = 8;
  while (2 * o.lanes * o.ts * o.tt <= OV_THREADS && 2 * o.lanes <= 32) o.lanes *= 2;
  return o;
}

// Chunks of a configuration's sites and their groups.  A lane's sums run over 64
// sites of a chunk (the tree and its share of the sums are then a tenth of the
// FMAs), over fewer in small volumes: a call waits for its longest CTA there, and 256
// threads a site apart, which were here before, had sums as short (32 of a
// lane's at N = 19 and L = 8 would have 1.7 times the error, rms).  At most 512
// chunks (the sums' buffer).
constexpr int OV_GROUPS = 8;
struct OvChunks {
  long sites;                       // of a chunk, a multiple of T
  int chunks, per_group, groups;
};
static OvChunks overlap_chunks(long vol, OvTile& o) {
  OvChunks c;
  c.sites = o.lanes * (vol <= 1024 ? 4 : vol <= 2048 ? 8 : vol <= 4096 ? 16 : vol <= 16384 ? 32 : 64);
  if (c.sites > 512) c.sites = 512;
  while ((vol + c.sites - 1) / c.sites > 512) c.sites *= 2;
  c.chunks = (int)((vol + c.sites - 1) / c.sites);
  c.per_group = (c.chunks + OV_GROUPS - 1) / OV_GROUPS;
  c.groups = (c.chunks + c.per_group - 1) / c.per_group;
  // stages: both buffers of two CTAs fit an SM up to 48 rows
  o.log_t = o.rows <= 8 ? 8 : o.rows <= 24 ? 7 : o.rows <= 48 ? 6 : 5;
  while ((1 << o.log_t) > c.sites) --o.log_t;
  o.T = 1 << o.log_t;
  return c;
}

// The end of a chunk: the tree over an entry's lanes, neighbours in one warp, which
// halve the N entries between them at each level while there are any to halve.
// Lane l is left with the sums of the entries from overlap_first<N>(l, lanes) on.
template <int N>
__device__ __forceinline__ void overlap_tree(double (&re)[N], double (&im)[N], int l, int lanes) {
  int off = lanes / 2;
#pragma unroll
  for (int h = N / 2; h >= 1; h >>= 1) {
    if (off == 0) continue;
    const bool up = l & off;
#pragma unroll
    for (int k = 0; k < h; ++k) {
      const double kr = up ? re[k + h] : re[k], sr = up ? re[k] : re[k + h];
      const double ki = up ? im[k + h] : im[k], si = up ? im[k] : im[k + h];
      re[k] = kr + __shfl_xor_sync(0xffffffffu, sr, off);
      im[k] = ki + __shfl_xor_sync(0xffffffffu, si, off);
    }
    off >>= 1;
  }
  for (; off > 0; off >>= 1) {
    re[0] += __shfl_xor_sync(0xffffffffu, re[0], off);
    im[0] += __shfl_xor_sync(0xffffffffu, im[0], off);
  }
}
template <int N>
__device__ __forceinline__ int overlap_first(int l, int lanes) {
  int e = 0, off = lanes / 2;
#pragma unroll
  for (int h = N / 2; h >= 1; h >>= 1, off >>= 1)
    if (l & off) e += h;
  return e;
}

// CTA r of the `ctas` of a configuration and tile takes chunks r per_cta .. ;
// each: every chunk's sums to out[conf][chunk], else out[conf] the whole sum (one
// CTA, or a cluster of one per group).
template <typename R>
__global__ void __launch_bounds__(OV_THREADS, 2) overlap_tile_kernel(const double2* __restrict__ src, int ns,
                                                                  const void* __restrict__ psi, int nt, int nconf,
                                                                  long vol, int ctas, int per_cta, int each,
                                                                  OvChunks ch, OvTile o, double* __restrict__ out) {
  extern __shared__ __align__(16) double2 ovs[];  // [2][rows][T], then [2][16 blocks]
  const int T = o.T, lanes = o.lanes;
  const long task = blockIdx.x / ctas;
  const int r = (int)(blockIdx.x - task * ctas);
  const long conf = task % nconf;
  const int tile = (int)(task / nconf);
  const int s0 = 4 * o.ts * (tile % o.ns_t), t0 = 4 * o.tt * (tile / o.ns_t);
  int chunk = r * per_cta;
  const int last = chunk + per_cta < ch.chunks ? chunk + per_cta : ch.chunks;
  const long p0 = chunk * ch.sites, p1 = last * ch.sites < vol ? last * ch.sites : vol;
  const cplx<R>* orb = reinterpret_cast<const cplx<R>*>(psi) + (size_t)conf * nt * vol;
  const int l = threadIdx.x % lanes, slot = threadIdx.x / lanes;
  const bool active = slot < o.ts * o.tt;
  const int bi = active ? slot / o.tt : 0, bj = active ? slot % o.tt : 0;
  auto fill = [&](long p, double2* t) {
    for (int e = threadIdx.x; e < o.rows * T; e += OV_THREADS) {
      const int row = e >> o.log_t;
      const long q = p + (e & (T - 1));
      const bool is_src = row < 4 * o.ts;
      const int i = is_src ? s0 + row : t0 + row - 4 * o.ts;
      if (q >= p1 || i >= (is_src ? ns : nt)) {
        t[e] = make_double2(0.0, 0.0);
      } else if (is_src || sizeof(R) == 8) {
        const void* g = is_src ? (const void*)(src + (size_t)i * vol + q) : (const void*)(orb + (size_t)i * vol + q);
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(t + e)), "l"(g)
                     : "memory");
      } else {  // FP32: into the element's upper half, spread by `widen`
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((uint32_t)__cvta_generic_to_shared(&t[e].y)),
                     "l"(orb + (size_t)i * vol + q)
                     : "memory");
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  // FP32 orbitals to FP64 in place, by the thread that copied them
  const int first = (int)threadIdx.x + 4 * o.ts * T / OV_THREADS * OV_THREADS;
  auto widen = [&](long p, double2* t) {
    for (int e = first; e < o.rows * T; e += OV_THREADS) {
      const int row = e >> o.log_t;
      const long q = p + (e & (T - 1));
      if (row >= 4 * o.ts && q < p1 && t0 + row - 4 * o.ts < nt) {
        const float2 v = *reinterpret_cast<const float2*>(&t[e].y);
        t[e] = make_double2((double)v.x, (double)v.y);
      }
    }
  };
  const int size = o.rows * T;
  // the sums of this thread's block: all groups', and the present one's
  double2* all = ovs + 2 * size + 16 * slot;
  double2* group = all + 16 * o.ts * o.tt;
  const int held = lanes == 8 ? 2 : 1;
  const bool owner = active && (lanes < 32 || l % 2 == 0);
  const int mine = overlap_first<16>(l, lanes);
  if (owner)
    for (int j = 0; j < held; ++j) all[mine + j] = group[mine + j] = make_double2(0.0, 0.0);
  double re[16], im[16];
#pragma unroll
  for (int k = 0; k < 16; ++k) re[k] = im[k] = 0.0;
  auto store = [&](size_t matrix, int k, double2 v) {
    const int s = s0 + 4 * bi + k / 4, t = t0 + 4 * bj + k % 4;
    if (s >= ns || t >= nt) return;
    double* to = out + 2 * ((matrix * ns + s) * nt + t);  // (the caller's S: on 8 bytes)
    to[0] = v.x;
    to[1] = v.y;
  };
  fill(p0, ovs);
  int buf = 0;
  for (long p = p0; p < p1; p += T, buf ^= 1) {
    __syncthreads();  // every thread is done with the buffer the next copies overwrite
    if (p + T < p1) fill(p + T, ovs + (buf ^ 1) * size);
    else asm volatile("cp.async.commit_group;" ::: "memory");
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    if (sizeof(R) == 4) widen(p, ovs + buf * size);
    __syncthreads();
    if (active) {
      const double2* ta = ovs + buf * size + 4 * bi * T;
      const double2* tb = ovs + buf * size + 4 * (o.ts + bj) * T;
      for (int q = l; q < T; q += lanes) {
        double2 b[4];
#pragma unroll
        for (int v = 0; v < 4; ++v) b[v] = tb[v * T + q];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const double2 a = ta[u * T + q];
#pragma unroll
          for (int v = 0; v < 4; ++v) {
            re[4 * u + v] = fma(a.x, b[v].x, re[4 * u + v]);
            im[4 * u + v] = fma(a.x, b[v].y, im[4 * u + v]);
          }
#pragma unroll
          for (int v = 0; v < 4; ++v) {
            re[4 * u + v] = fma(a.y, b[v].y, re[4 * u + v]);
            im[4 * u + v] = fma(-a.y, b[v].x, im[4 * u + v]);
          }
        }
      }
    }
    if (p + T < p1 && p + T < (chunk + 1) * ch.sites) continue;
    overlap_tree(re, im, l, lanes);
    const bool closes = (chunk + 1) % ch.per_group == 0 || chunk + 1 == ch.chunks;
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      if (!owner || j >= held) continue;
      const double2 v = make_double2(re[j], im[j]);
      if (each) {
        store((size_t)conf * ch.chunks + chunk, mine + j, v);
      } else {
        double2 g = group[mine + j];
        g.x += v.x;
        g.y += v.y;
        if (closes) {
          all[mine + j].x += g.x;
          all[mine + j].y += g.y;
          g = make_double2(0.0, 0.0);
        }
        group[mine + j] = g;
      }
    }
#pragma unroll
    for (int k = 0; k < 16; ++k) re[k] = im[k] = 0.0;
    ++chunk;
  }
  if (each) return;
  if (ctas == 1) {
    if (owner)
      for (int j = 0; j < held; ++j) store(conf, mine + j, all[mine + j]);
    return;
  }
  // a cluster holds the groups of its configuration: entries spread over its CTAs
  cg::cluster_group cluster = cg::this_cluster();
  cluster.sync();
  for (int e = r * OV_THREADS + threadIdx.x; e < 16 * o.ts * o.tt; e += ctas * OV_THREADS) {
    double2 v = make_double2(0.0, 0.0);
    for (int g = 0; g < ctas; ++g) {
      const double2 w = cluster.map_shared_rank(ovs + 2 * size, g)[e];
      v.x += w.x;
      v.y += w.y;
    }
    const int b = e / 16, s = s0 + 4 * (b / o.tt) + e % 16 / 4, t = t0 + 4 * (b % o.tt) + e % 4;
    if (s < ns && t < nt) {
      double* to = out + 2 * (((size_t)conf * ns + s) * nt + t);
      to[0] = v.x;
      to[1] = v.y;
    }
  }
  cluster.sync();  // peers keep their shared memory until every sum is read
}

// The same sums without staging: LANES lanes take one orbital and one group of its
// chunks, NX sources (blockIdx.y's) in registers; the groups of an orbital meet
// in shared memory.  With few sources or orbitals there is little to reuse, the
// orbitals are the traffic, and the tile kernel keeps too few bytes in flight (a
// 4 x 4 block mostly padding on top); in small calls its chain is the shorter one.
// FP64, N = 2, 200 configurations at L = 32: 47 us against 285 by tiles (a block
// per orbital: 87); 19 sources and one orbital, L = 16, 1500 configurations 150
// against 510 (148); N = 9, L = 8, one configuration 12 against 17 (12).  Four sites
// in flight per lane: two cost 13 % in the mean over N = 1 .. 33, L = 8 .. 48.  As many
// sources as there are: groups of eight with the rest masked took 7 % more (N = 10,
// L = 12, 512 configurations 210 us, now 146).
constexpr int OD_WARPS = 8;

// Sources of a group: near-equal groups of at most eight
constexpr int overlap_direct_sources(int ns) {
  return ns <= 2 ? 2 : ns <= 4 ? 4 : (ns + (ns + 7) / 8 - 1) / ((ns + 7) / 8);
}

template <typename R, int NX, int LANES, bool MANY>
__global__ void __launch_bounds__(32 * OD_WARPS, NX <= 4 || MANY ? 3 : 2)
    overlap_direct_kernel(const double2* __restrict__ src, int ns, const void* __restrict__ psi, int nt, long vol,
                          long orbitals, OvChunks ch, double* __restrict__ S) {
  constexpr int SUB = 32 / LANES, SB = NX <= 2 ? 2 : NX <= 4 ? 4 : 8;  // orbitals of a warp, entries of the tree
  constexpr int UNROLL = MANY ? 2 : 4;
  __shared__ double2 sums[OD_WARPS][SUB][SB];
  const int l = threadIdx.x % LANES, sub = threadIdx.x % 32 / LANES, warp = threadIdx.x >> 5;
  const int s0 = NX * (int)blockIdx.y, sb = ns - s0 < NX ? ns - s0 : NX;
  const double2* from = src + (size_t)s0 * vol;
  const int here = OD_WARPS / ch.groups, g = warp % ch.groups;  // warps per group of this CTA, the warp's group
  const long first = (long)blockIdx.x * here * SUB, orbital = first + warp / ch.groups * SUB + sub;
  const bool active = warp < here * ch.groups && orbital < orbitals;
  const cplx<R>* orb = reinterpret_cast<const cplx<R>*>(psi) + (size_t)(active ? orbital : 0) * vol;
  double gr = 0.0, gi = 0.0;
  // (a warp's lanes go through the same chunks: the tree's shuffles are the warp's)
  const int end_chunk = (g + 1) * ch.per_group < ch.chunks ? (g + 1) * ch.per_group : ch.chunks;
  const int last = warp < here * ch.groups ? end_chunk : 0;
  for (int chunk = g * ch.per_group; chunk < last; ++chunk) {
    double re[SB], im[SB];
#pragma unroll
    for (int k = 0; k < SB; ++k) re[k] = im[k] = 0.0;
    const long end = (chunk + 1) * ch.sites < vol ? (chunk + 1) * ch.sites : vol;
#pragma unroll UNROLL
    for (long q = chunk * ch.sites + l; q < end; q += LANES) {
      const cplx<R> v = orb[q];
      const double br = (double)v.re, bi = (double)v.im;
      double2 a[NX];
#pragma unroll
      for (int u = 0; u < NX; ++u) a[u] = u < sb ? __ldg(from + (size_t)u * vol + q) : make_double2(0.0, 0.0);
#pragma unroll
      for (int u = 0; u < NX; ++u) {
        re[u] = fma(a[u].x, br, re[u]);
        im[u] = fma(a[u].x, bi, im[u]);
        re[u] = fma(a[u].y, bi, re[u]);
        im[u] = fma(-a[u].y, br, im[u]);
      }
    }
    overlap_tree<SB>(re, im, l, LANES);
    gr += re[0];
    gi += im[0];
  }
  if (l % (LANES / SB) == 0) sums[warp][sub][overlap_first<SB>(l, LANES)] = make_double2(gr, gi);
  __syncthreads();
  for (int e = threadIdx.x; e < here * SUB * SB; e += 32 * OD_WARPS) {
    const int s = e % SB, k = e / SB;  // orbital first + k
    if (s >= sb || first + k >= orbitals) continue;
    double2 v = make_double2(0.0, 0.0);
    for (int i = 0; i < ch.groups; ++i) {
      const double2 w = sums[k / SUB * ch.groups + i][k % SUB][s];
      v.x += w.x;
      v.y += w.y;
    }
    const long conf = (first + k) / nt, t = (first + k) % nt;
    double* to = S + 2 * ((conf * ns + s0 + s) * nt + t);
    to[0] = v.x;
    to[1] = v.y;
  }
}

// S[c][e] = the chunks' sums, group by group; sixteen loads in flight (one by one
// the 64 chunks of a single configuration, N = 19, L = 32, took 19.5 us; now
// 10.0).
__global__ void overlap_sum_kernel(const double2* __restrict__ part, OvChunks ch, long per_conf, long total,
                                   double* __restrict__ S) {
  for (long e = (long)blockIdx.x * blockDim.x + threadIdx.x; e < total; e += (long)gridDim.x * blockDim.x) {
    const long c = e / per_conf, i = e - c * per_conf;
    const double2* p = part + (size_t)c * ch.chunks * per_conf + i;
    double2 v = make_double2(0.0, 0.0), group = v;
    int left = ch.per_group;  // chunks to come of the present group
    for (int k0 = 0; k0 < ch.chunks; k0 += 16) {
      double2 w[16];
#pragma unroll
      for (int k = 0; k < 16; ++k)
        if (k0 + k < ch.chunks) w[k] = __ldcg(p + (size_t)(k0 + k) * per_conf);
#pragma unroll
      for (int k = 0; k < 16; ++k)
        if (k0 + k < ch.chunks) {
          group.x += w[k].x;
          group.y += w[k].y;
          if (--left == 0 || k0 + k + 1 == ch.chunks) {
            v.x += group.x;
            v.y += group.y;
            group = make_double2(0.0, 0.0);
            left = ch.per_group;
          }
        }
    }
    S[2 * e] = v.x;
    S[2 * e + 1] = v.y;
  }
}

// Plane-wave sources: S[c][s][t] = psi_{c,t}(p_s) exactly.
template <typename R>
__global__ void gather_kernel(const int* __restrict__ index, int ns, const void* __restrict__ psi, int nt,
                              int nconf, long vol, double* __restrict__ S) {
  long total = (long)nconf * ns * nt;
  for (long e = (long)blockIdx.x * blockDim.x + threadIdx.x; e < total; e += (long)gridDim.x * blockDim.x) {
    long conf = e / ((long)ns * nt);
    int s = (int)((e / nt) % ns), t = (int)(e % nt);
    const int p = index[s];
    // a lattice index outside [0, vol) has no overlap with the orbitals
    cplx<R> q = (p >= 0 && p < vol) ? ld<R>(psi, ((conf * nt + t) * vol) + p) : cplx<R>{(R)0, (R)0};
    S[2 * e] = (double)q.re;
    S[2 * e + 1] = (double)q.im;
  }
}

// ------------------------------------------------------------ pair matrix
// One block per (configuration, s, t): phi = sum_i w_i psi1_s(i) psi2_t(opp(i)).
template <typename R>
__global__ void __launch_bounds__(256) pair_kernel(const void* __restrict__ psi1, const void* __restrict__ psi2,
                                                   int n, long vol, const double* __restrict__ w,
                                                   const int* __restrict__ opp, double* __restrict__ phi) {
  const long e = blockIdx.x;  // (conf * n + s) * n + t
  const long conf = e / ((long)n * n);
  const int s = (int)((e / n) % n), t = (int)(e % n);
  const char* a = reinterpret_cast<const char*>(psi1) + (size_t)(conf * n + s) * vol * 2 * sizeof(R);
  const char* b = reinterpret_cast<const char*>(psi2) + (size_t)(conf * n + t) * vol * 2 * sizeof(R);
  double re = 0.0, im = 0.0;
  for (long i = threadIdx.x; i < vol; i += blockDim.x) {
    const int j = opp[i];
    if (j < 0 || j >= vol) continue;  // a partner outside the lattice contributes nothing
    cplx<R> x = ld<R>(a, i), y = ld<R>(b, j);
    double wi = w[i];
    re += ((double)x.re * y.re - (double)x.im * y.im) * wi;
    im += ((double)x.re * y.im + (double)x.im * y.re) * wi;
  }
  __shared__ double red[2][8];
  for (int off = 16; off > 0; off >>= 1) {
    re += __shfl_down_sync(0xffffffffu, re, off);
    im += __shfl_down_sync(0xffffffffu, im, off);
  }
  if ((threadIdx.x & 31) == 0) {
    red[0][threadIdx.x >> 5] = re;
    red[1][threadIdx.x >> 5] = im;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double sr = 0, si = 0;
    for (int k = 0; k < (int)(blockDim.x >> 5); ++k) {
      sr += red[0][k];
      si += red[1][k];
    }
    phi[2 * e] = sr;
    phi[2 * e + 1] = si;
  }
}

// Tiled pair matrices for n <= 32 (the path of nrcps_pair_matrix and of the
// ensemble's pair sink).  One thread-block cluster of up to eight CTAs per
// configuration; CTA r of C takes every C-th tile of ts sites.
//
// TwoBody's opposite-parity index is an involution (opp(opp(i)) = i), so the
// sites pair up: a tile stages, for every site i of the tile with i <= opp(i),
// the term of i, a_s = w_i psi1_s(i) and b_t = psi2_t(opp(i)), and (when
// i < opp(i)) the term of j = opp(i), a_s = w_j psi1_s(j) and b_t = psi2_t(i).
// Every term is summed exactly once and every orbital element is read once
// (the gathered rows are the rows the pair's other term reads directly);
// tiles whose sites all have i > opp(i) are skipped after reading opp.  When
// `bad_opp` points at a nonzero word (the table is not an involution) the
// tiles stage the term of every site instead: the plain gather.
//
// Thread (block, group) accumulates a 2 x 2 block of phi over the group's
// slots of every tile, in R within a tile and in FP64 across tiles; the
// groups are summed in shared memory and the cluster's CTAs in rank order
// through distributed shared memory: the result does not depend on timing.
//
// With psi1 = psi2 and a weight even under the pairing (w(opp(i)) = w(i),
// TwoBody's tables), the pair of terms of i and opp(i) is symmetric in
// (s, t), so phi is: only the blocks on and above the diagonal are summed
// and each is written to both triangles (FP32 orbitals with n = 9 .. 20 mostly
// take pair_sym.cu instead).
constexpr int PAIR_THREADS = 256;
constexpr int PAIR_MAXN = 32;
constexpr int PB = 2;                // register block: PB x PB complex pair-matrix entries per thread
constexpr int PAIR_E = PB * PB * 2;  // doubles per block

template <typename R>
struct PairShape {
  static int rows(int n) { return (n + PB - 1) / PB * PB; }  // staged rows, padded to whole blocks
  // sites per tile: at most about 20 KB of staged rows per array (four CTAs per SM)
  static int ts(int n) {
    const int budget = (sizeof(R) == 4 ? 1280 : 640) / rows(n);
    int t = 16;
    while (t * 2 <= budget && t < 128) t *= 2;
    return t;
  }
  static int ld(int n) { return 2 * ts(n) + 1; }  // slots per staged row, padded: rows start in different banks
  static size_t smem(int n) {
    const size_t t = 2 * (size_t)rows(n) * ld(n) * sizeof(cplx<R>);
    const size_t nb = rows(n) / PB, red = nb * nb * PAIR_E * sizeof(double);
    return t > red ? t : red;
  }
};

// Block blk of the upper triangle (row-major, bi <= bj) or of the full
// nb x nb grid
__device__ __forceinline__ void pair_block(int blk, int nb, bool sym, int& bi, int& bj) {
  if (!sym) {
    bi = blk / nb;
    bj = blk % nb;
    return;
  }
  bi = 0;
  while (blk >= nb - bi) {
    blk -= nb - bi;
    ++bi;
  }
  bj = bi + blk;
}

// The end of a tiled pair kernel: the groups of every block summed in shared
// memory (fixed order), then the cluster's CTAs in rank order through
// distributed shared memory, written by rank 0 (to both triangles for the
// symmetric form).
__device__ __forceinline__ void pair_reduce_store(const double (&acc)[PB][PB][2], unsigned char* smem, int n,
                                                  int nb, bool sym, int nblk, int groups, int g, int blk,
                                                  bool active, long conf, double* __restrict__ phi) {
  cg::cluster_group cluster = cg::this_cluster();
  const int split = (int)cluster.num_blocks(), rank = (int)cluster.block_rank();
  __syncthreads();
  double* red = reinterpret_cast<double*>(smem);  // [nblk][PAIR_E], over the staged tiles
  for (int gg = 0; gg < groups; ++gg) {
    if (active && g == gg) {
#pragma unroll
      for (int a = 0; a < PB; ++a)
#pragma unroll
        for (int b = 0; b < PB; ++b)
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            const int e = blk * PAIR_E + (a * PB + b) * 2 + c;
            red[e] = (gg == 0 ? 0.0 : red[e]) + acc[a][b][c];
          }
    }
    __syncthreads();
  }
  cluster.sync();  // every CTA's sums are in its shared memory
  if (rank == 0) {
    for (int e = threadIdx.x; e < nblk * PAIR_E; e += PAIR_THREADS) {
      double v = 0.0;
      for (int r2 = 0; r2 < split; ++r2) v += cluster.map_shared_rank(red, r2)[e];
      const int k = e % PAIR_E;
      int bi, bj;
      pair_block(e / PAIR_E, nb, sym, bi, bj);
      const int s = PB * bi + (k / 2) / PB, t = PB * bj + (k / 2) % PB;
      // (the symmetric form writes each entry with s <= t to both places)
      if (s < n && t < n && (!sym || s <= t)) {
        phi[2 * ((conf * n + s) * (long)n + t) + (k & 1)] = v;
        if (sym && s != t) phi[2 * ((conf * n + t) * (long)n + s) + (k & 1)] = v;
      }
    }
  }
  cluster.sync();  // peers keep their shared memory until rank 0 has read it
}

template <typename R>
__global__ void __launch_bounds__(PAIR_THREADS, 4)
    pair_tile_kernel(const void* __restrict__ psi1, const void* __restrict__ psi2, int n, long vol,
                     const double* __restrict__ w, const int* __restrict__ opp, const int* __restrict__ flags,
                     int host_flags, int leave_sym, int ts, double* __restrict__ phi) {
  if (leave_sym && !*flags) return;  // pair_sym_kernel's
  extern __shared__ __align__(16) unsigned char pair_smem[];
  const int LD = 2 * ts + 1;
  const int nb = (n + PB - 1) / PB, rows = nb * PB;
  cplx<R>* A = reinterpret_cast<cplx<R>*>(pair_smem);  // [rows][LD]: w psi1 of each slot's term
  cplx<R>* B = A + (size_t)rows * LD;                   // [rows][LD]: psi2 at the term's partner site
  cg::cluster_group cluster = cg::this_cluster();
  const int split = (int)cluster.num_blocks(), rank = (int)cluster.block_rank();
  const long conf = blockIdx.x / split;
  const cplx<R>* p1 = reinterpret_cast<const cplx<R>*>(psi1) + (size_t)conf * n * vol;
  const cplx<R>* p2 = reinterpret_cast<const cplx<R>*>(psi2) + (size_t)conf * n * vol;
  // the table's properties: bit 0 opp is no involution, bit 1 w is not even
  // under opp (from the device check when there is one)
  const int fl = flags ? *flags : host_flags;
  const bool paired = !(fl & 1);
  const bool sym = paired && !(fl & 2) && psi1 == psi2;
  // staging: thread -> (slot q of the tile, orbital lane)
  const int q = threadIdx.x % ts, olane = threadIdx.x / ts, ostride = PAIR_THREADS / ts;
  // accumulation: thread -> (PB x PB block, group), blocks fastest: the
  // lanes of a warp read one slot of at most 2 nb rows, in distinct banks
  const int nblk = sym ? nb * (nb + 1) / 2 : nb * nb;
  const int groups = PAIR_THREADS / nblk;  // >= 1 for n <= 32
  const int g = threadIdx.x / nblk, blk = threadIdx.x % nblk;
  const bool active = g < groups;
  int bi = 0, bj = 0;
  if (active) pair_block(blk, nb, sym, bi, bj);
  const int abase = bi * PB * LD, bbase = bj * PB * LD;
  for (int e = threadIdx.x; e < (rows - n) * LD; e += PAIR_THREADS) {  // the padding row stays zero
    A[n * LD + e] = cplx<R>{(R)0, (R)0};
    B[n * LD + e] = cplx<R>{(R)0, (R)0};
  }
  double acc[PB][PB][2];
#pragma unroll
  for (int a = 0; a < PB; ++a)
#pragma unroll
    for (int b = 0; b < PB; ++b) acc[a][b][0] = acc[a][b][1] = 0.0;
  const long ntiles = (vol + ts - 1) / ts;
  for (long tile = rank; tile < ntiles; tile += split) {
    const long i = tile * ts + q;
    const bool valid = i < vol;
    const long j = valid ? (long)__ldg(opp + i) : 0;
    // (the plain gather skips a partner outside the lattice; a paired table
    // has none)
    const bool take = valid && (paired ? i <= j : (j >= 0 && j < vol));
    const bool second = paired && valid && i < j;
    // also the barrier after the previous tile's accumulation
    if (!__syncthreads_or(take)) continue;
    const R wi = take ? (R)__ldg(w + i) : (R)0, wj = second ? (R)__ldg(w + j) : (R)0;
#pragma unroll 4
    for (int o = olane; o < n; o += ostride) {
      const cplx<R>* r1 = p1 + (size_t)o * vol;
      const cplx<R>* r2 = p2 + (size_t)o * vol;
      cplx<R> a1{(R)0, (R)0}, b1{(R)0, (R)0}, a2{(R)0, (R)0}, b2{(R)0, (R)0};
      if (take) {
        a1 = r1[i];
        b1 = r2[j];
      }
      if (second) {
        a2 = r1[j];
        b2 = r2[i];
      }
      A[o * LD + q] = cplx<R>{a1.re * wi, a1.im * wi};
      B[o * LD + q] = b1;
      A[o * LD + ts + q] = cplx<R>{a2.re * wj, a2.im * wj};
      B[o * LD + ts + q] = b2;
    }
    __syncthreads();
    if (active) {
      // sum over the slots of a_s b_t (complex, no conjugation) in R: two
      // fused multiply-adds per real component; then into the FP64 sums
      R r[PB][PB][2];
#pragma unroll
      for (int a = 0; a < PB; ++a)
#pragma unroll
        for (int b = 0; b < PB; ++b) r[a][b][0] = r[a][b][1] = (R)0;
      for (int slot = g; slot < 2 * ts; slot += groups) {
        cplx<R> av[PB], bv[PB];
#pragma unroll
        for (int k = 0; k < PB; ++k) {
          av[k] = A[abase + k * LD + slot];
          bv[k] = B[bbase + k * LD + slot];
        }
#pragma unroll
        for (int a = 0; a < PB; ++a)
#pragma unroll
          for (int b = 0; b < PB; ++b) {
            r[a][b][0] = fma(av[a].re, bv[b].re, r[a][b][0]);
            r[a][b][0] = fma(-av[a].im, bv[b].im, r[a][b][0]);
            r[a][b][1] = fma(av[a].re, bv[b].im, r[a][b][1]);
            r[a][b][1] = fma(av[a].im, bv[b].re, r[a][b][1]);
          }
      }
#pragma unroll
      for (int a = 0; a < PB; ++a)
#pragma unroll
        for (int b = 0; b < PB; ++b) {
          acc[a][b][0] += (double)r[a][b][0];
          acc[a][b][1] += (double)r[a][b][1];
        }
    }
  }
  pair_reduce_store(acc, pair_smem, n, nb, sym, nblk, groups, g, blk, active, conf, phi);
}

// *flags |= 1 unless opp is an involution of [0, vol) (TwoBody's parity
// mirror is), |= 2 unless w(opp(i)) = w(i) for every i
__global__ void opp_involution_check_kernel(const int* __restrict__ opp, const double* __restrict__ w, long vol,
                                            int* flags) {
  for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < vol; i += (long)gridDim.x * blockDim.x) {
    const int j = opp[i];
    if (j < 0 || j >= vol) {
      atomicOr(flags, 3);
    } else {
      if (opp[j] != i) atomicOr(flags, 1);
      if (w[j] != w[i]) atomicOr(flags, 2);
    }
  }
}

// GeneralizedTwoBody::Run (src/two_body/noarch/two_body_run.C:45-75) batched:
// phi[c][s][t] = sum_l sum_i wl[l][i] psi1_{c,s}(shift[l][i]) psi2_{c,t}(opp(i))
// with wl[l][i] = weight(R, l) * half_site_wavefunc[l][i] folded by the
// caller.  One block per (conf, s, t); the term loop is outermost, as in the
// reference.
template <typename R>
__global__ void __launch_bounds__(256) shifted_pair_kernel(const void* __restrict__ psi1,
                                                           const void* __restrict__ psi2, int n, long vol, int nterms,
                                                           const int* __restrict__ shift,
                                                           const double* __restrict__ wl,
                                                           const int* __restrict__ opp, double* __restrict__ phi) {
  const long e = blockIdx.x;  // (conf * n + s) * n + t
  const long conf = e / ((long)n * n);
  const int s = (int)((e / n) % n), t = (int)(e % n);
  const char* a = reinterpret_cast<const char*>(psi1) + (size_t)(conf * n + s) * vol * 2 * sizeof(R);
  const char* b = reinterpret_cast<const char*>(psi2) + (size_t)(conf * n + t) * vol * 2 * sizeof(R);
  double re = 0.0, im = 0.0;
  for (int l = 0; l < nterms; ++l) {
    const int* sh = shift + (size_t)l * vol;
    const double* w = wl + (size_t)l * vol;
    for (long i = threadIdx.x; i < vol; i += blockDim.x) {
      const int si = sh[i], j = opp[i];
      if (si < 0 || si >= vol || j < 0 || j >= vol) continue;  // outside the lattice: no term
      cplx<R> x = ld<R>(a, si), y = ld<R>(b, j);
      const double wi = w[i];
      re += ((double)x.re * y.re - (double)x.im * y.im) * wi;
      im += ((double)x.re * y.im + (double)x.im * y.re) * wi;
    }
  }
  __shared__ double red[2][8];
  for (int off = 16; off > 0; off >>= 1) {
    re += __shfl_down_sync(0xffffffffu, re, off);
    im += __shfl_down_sync(0xffffffffu, im, off);
  }
  if ((threadIdx.x & 31) == 0) {
    red[0][threadIdx.x >> 5] = re;
    red[1][threadIdx.x >> 5] = im;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double sr = 0, si = 0;
    for (int k = 0; k < (int)(blockDim.x >> 5); ++k) {
      sr += red[0][k];
      si += red[1][k];
    }
    phi[2 * e] = sr;
    phi[2 * e + 1] = si;
  }
}

// ------------------------------------------------- pointer-array variants
// mat[t + nf*s] = <kets[s] | bras[t]> (the layout of Cuda::InnerProduct,
// src/utils/cuda/cuda_utils_kernels.cu:4-48), FP64, one block per (s, t).
__global__ void __launch_bounds__(256) inner_ptrs_kernel(const double* const* __restrict__ kets,
                                                         const double* const* __restrict__ bras, int nf, long vol,
                                                         double* __restrict__ mat) {
  const int s = blockIdx.x / nf, t = blockIdx.x % nf;
  const double2* a = reinterpret_cast<const double2*>(kets[s]);
  const double2* b = reinterpret_cast<const double2*>(bras[t]);
  double re = 0.0, im = 0.0;
  for (long i = threadIdx.x; i < vol; i += blockDim.x) {
    double2 x = a[i], y = b[i];
    re = fma(x.x, y.x, re);
    re = fma(x.y, y.y, re);
    im = fma(x.x, y.y, im);
    im = fma(-x.y, y.x, im);
  }
  __shared__ double red[2][8];
  for (int o = 16; o > 0; o >>= 1) {
    re += __shfl_down_sync(0xffffffffu, re, o);
    im += __shfl_down_sync(0xffffffffu, im, o);
  }
  if ((threadIdx.x & 31) == 0) {
    red[0][threadIdx.x >> 5] = re;
    red[1][threadIdx.x >> 5] = im;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double sr = 0, si = 0;
    for (int k = 0; k < (int)(blockDim.x >> 5); ++k) {
      sr += red[0][k];
      si += red[1][k];
    }
    mat[2L * (t + (long)nf * s)] = sr;
    mat[2L * (t + (long)nf * s) + 1] = si;
  }
}

// phi[t + nf*s] = sum_i w_i props1[s](i) props2[t](opp(i)), FP64.
__global__ void __launch_bounds__(256) pair_ptrs_kernel(const double* const* __restrict__ p1,
                                                        const double* const* __restrict__ p2, int nf, long vol,
                                                        const double* __restrict__ w, const int* __restrict__ opp,
                                                        double* __restrict__ phi) {
  const int s = blockIdx.x / nf, t = blockIdx.x % nf;
  const double2* a = reinterpret_cast<const double2*>(p1[s]);
  const double2* b = reinterpret_cast<const double2*>(p2[t]);
  double re = 0.0, im = 0.0;
  for (long i = threadIdx.x; i < vol; i += blockDim.x) {
    double2 x = a[i], y = b[opp[i]];
    const double wi = w[i];
    re += (x.x * y.x - x.y * y.y) * wi;
    im += (x.x * y.y + x.y * y.x) * wi;
  }
  __shared__ double red[2][8];
  for (int o = 16; o > 0; o >>= 1) {
    re += __shfl_down_sync(0xffffffffu, re, o);
    im += __shfl_down_sync(0xffffffffu, im, o);
  }
  if ((threadIdx.x & 31) == 0) {
    red[0][threadIdx.x >> 5] = re;
    red[1][threadIdx.x >> 5] = im;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double sr = 0, si = 0;
    for (int k = 0; k < (int)(blockDim.x >> 5); ++k) {
      sr += red[0][k];
      si += red[1][k];
    }
    phi[2L * (t + (long)nf * s)] = sr;
    phi[2L * (t + (long)nf * s) + 1] = si;
  }
}

// ------------------------------------------------------------------- LU
struct dc {
  double re, im;
};
__device__ __forceinline__ dc dmul(dc a, dc b) { return dc{a.re * b.re - a.im * b.im, a.re * b.im + a.im * b.re}; }
__device__ __forceinline__ double dabs(dc a) { return hypot(a.re, a.im); }
__device__ __forceinline__ dc drecip(dc b) {
  // 1 / b with Smith's scaling
  if (fabs(b.re) >= fabs(b.im)) {
    double r = b.im / b.re, d = b.re + b.im * r;
    return dc{1.0 / d, -r / d};
  }
  double r = b.re / b.im, d = b.re * r + b.im;
  return dc{r / d, -1.0 / d};
}

// Crout LU with implicit-scaled partial pivoting (src/utils/ludcmp.C:9-65)
// on the n x n matrix a (row-major, stride n).  Returns the permutation
// parity d, or 0 when a row is all zero (the reference exits there).
__device__ double ludcmp_dev(dc* a, int n, double* vv) {
  double d = 1.0;
  for (int i = 0; i < n; ++i) {
    double big = 0.0;
    for (int j = 0; j < n; ++j) {
      double t = dabs(a[n * i + j]);
      if (t > big) big = t;
    }
    if (big == 0.0) return 0.0;
    vv[i] = 1.0 / big;
  }
  int imax = 0;
  for (int j = 0; j < n; ++j) {
    for (int i = 0; i < j; ++i) {
      dc sum = a[n * i + j];
      for (int k = 0; k < i; ++k) {
        dc p = dmul(a[n * i + k], a[n * k + j]);
        sum.re -= p.re;
        sum.im -= p.im;
      }
      a[n * i + j] = sum;
    }
    double big = 0.0;
    for (int i = j; i < n; ++i) {
      dc sum = a[n * i + j];
      for (int k = 0; k < j; ++k) {
        dc p = dmul(a[n * i + k], a[n * k + j]);
        sum.re -= p.re;
        sum.im -= p.im;
      }
      a[n * i + j] = sum;
      double dum = vv[i] * dabs(sum);
      if (dum >= big) {
        big = dum;
        imax = i;
      }
    }
    if (j != imax) {
      for (int k = 0; k < n; ++k) {
        dc t = a[n * imax + k];
        a[n * imax + k] = a[n * j + k];
        a[n * j + k] = t;
      }
      d = -d;
      vv[imax] = vv[j];
    }
    if (dabs(a[n * j + j]) == 0.0) a[n * j + j] = dc{1.0e-20, 0.0};
    dc r = drecip(a[n * j + j]);
    for (int i = j + 1; i < n; ++i) a[n * i + j] = dmul(a[n * i + j], r);
  }
  return d;
}

// One thread per (matrix, measured minor).  Scratch: per thread n*n complex
// + n doubles in global memory (L2-resident).
__global__ void slater_dets_kernel(const double* __restrict__ S, const double* __restrict__ psi1, int N, int nconf,
                                   int mode, int log_det, double* __restrict__ out, double* scratch,
                                   long out_conf_stride, long out_offset) {
  const int nmeas = mode ? 2 * N : N;
  const long total = (long)nconf * nmeas;
  for (long e = (long)blockIdx.x * blockDim.x + threadIdx.x; e < total; e += (long)gridDim.x * blockDim.x) {
    const long c = e / nmeas;
    const int m = (int)(e % nmeas);
    const int n = mode ? m / 2 + 1 : m + 1;
    const int t0 = (mode && (m % 2 == 0)) ? n - 1 : -1;
    dc* a = reinterpret_cast<dc*>(scratch + e * (2L * N * N + N));
    double* vv = scratch + e * (2L * N * N + N) + 2L * N * N;
    const dc* Sc = reinterpret_cast<const dc*>(S) + c * (long)N * N;
    for (int i = 0; i < n; ++i)
      for (int j = 0; j < n; ++j) a[n * i + j] = Sc[(long)N * i + j];
    if (t0 >= 0) {
      // SlaterDet2::Run column t0 from psi1[s + t0*N] (slater_det2.C:102-106)
      const dc* P = reinterpret_cast<const dc*>(psi1) + c * (long)N * N;
      for (int i = 0; i < n; ++i) a[n * i + t0] = P[i + (long)t0 * N];
    }
    double d = ludcmp_dev(a, n, vv);
    dc r;
    if (!log_det) {
      r = dc{d, 0.0};
      for (int i = 0; i < n; ++i) r = dmul(r, a[n * i + i]);
    } else {
      // log(d) + sum log(U_ii), principal branches (slater_det.C:102-109)
      r = dc{log(fabs(d)), d < 0 ? 3.14159265358979323846 : 0.0};
      for (int i = 0; i < n; ++i) {
        r.re += log(dabs(a[n * i + i]));
        r.im += atan2(a[n * i + i].im, a[n * i + i].re);
      }
    }
    if (d == 0.0) r = dc{nan(""), nan("")};  // singular: flagged to the host
    double* o = out + c * out_conf_stride + out_offset + 2L * m;
    o[0] = r.re;
    o[1] = r.im;
  }
}

// One warp per (matrix, measured minor), the minor in shared memory.  The
// same Crout factorisation with implicit-scaled partial pivoting as
// ludcmp_dev, organised right-looking: element (i, k) receives the products
// l_ij u_jk in the same order j = 0, 1, ... as Crout's running sum, the
// pivot search sees the same updated column, ties go to the last row as
// in `if (dum >= big)`, and rows swap whole -- so the factors and the
// determinant follow the same arithmetic.  Lanes split rows (pivot search,
// multipliers) and columns (swaps, trailing update); no global scratch.
constexpr int kWarpLuMaxWarps = 4;  // warps per block (fewer for large N: shared memory)

__global__ void __launch_bounds__(32 * kWarpLuMaxWarps) slater_dets_warp_kernel(const double* __restrict__ S,
                                                                            const double* __restrict__ psi1, int N,
                                                                            int nconf, int mode, int log_det,
                                                                            double* __restrict__ out,
                                                                            long out_conf_stride, long out_offset) {
  extern __shared__ __align__(16) unsigned char lu_smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int wpb = blockDim.x >> 5;
  dc* a = reinterpret_cast<dc*>(lu_smem) + (size_t)warp * N * N;
  double* vv = reinterpret_cast<double*>(reinterpret_cast<dc*>(lu_smem) + (size_t)wpb * N * N) + warp * N;
  const int nmeas = mode ? 2 * N : N;
  const long total = (long)nconf * nmeas;
  for (long e = (long)blockIdx.x * wpb + warp; e < total; e += (long)gridDim.x * wpb) {
    const long c = e / nmeas;
    const int m = (int)(e % nmeas);
    const int n = mode ? m / 2 + 1 : m + 1;
    const int t0 = (mode && (m % 2 == 0)) ? n - 1 : -1;
    const dc* Sc = reinterpret_cast<const dc*>(S) + c * (long)N * N;
    const dc* P = mode ? reinterpret_cast<const dc*>(psi1) + c * (long)N * N : nullptr;
    for (int idx = lane; idx < n * n; idx += 32) {
      const int i = idx / n, k = idx - i * n;
      // SlaterDet2::Run column t0 from psi1[s + t0*N] (slater_det2.C:102-106)
      a[idx] = (k == t0) ? P[i + (long)t0 * N] : Sc[(long)N * i + k];
    }
    __syncwarp();
    bool zero_row = false;
    for (int i = lane; i < n; i += 32) {
      double big = 0.0;
      for (int k = 0; k < n; ++k) big = fmax(big, dabs(a[n * i + k]));
      if (big == 0.0) zero_row = true;
      vv[i] = 1.0 / big;
    }
    const bool singular = __any_sync(0xffffffffu, zero_row);
    __syncwarp();
    double d = 1.0;
    for (int j = 0; j < n && !singular; ++j) {
      double best = -1.0;
      int bi = -1;
      for (int i = j + lane; i < n; i += 32) {
        const double dum = vv[i] * dabs(a[n * i + j]);
        if (dum >= best) {
          best = dum;
          bi = i;
        }
      }
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) {
        const double ob = __shfl_xor_sync(0xffffffffu, best, off);
        const int oi = __shfl_xor_sync(0xffffffffu, bi, off);
        if (ob > best || (ob == best && oi > bi)) {
          best = ob;
          bi = oi;
        }
      }
      const int imax = bi;
      if (imax != j) {
        for (int k = lane; k < n; k += 32) {
          const dc t = a[n * imax + k];
          a[n * imax + k] = a[n * j + k];
          a[n * j + k] = t;
        }
        d = -d;
        if (lane == 0) vv[imax] = vv[j];
      }
      __syncwarp();
      if (lane == 0 && dabs(a[n * j + j]) == 0.0) a[n * j + j] = dc{1.0e-20, 0.0};
      __syncwarp();
      const dc r = drecip(a[n * j + j]);
      for (int i = j + 1 + lane; i < n; i += 32) a[n * i + j] = dmul(a[n * i + j], r);
      __syncwarp();
      for (int k = j + 1 + lane; k < n; k += 32) {
        const dc u = a[n * j + k];
        for (int i = j + 1; i < n; ++i) {
          const dc p = dmul(a[n * i + j], u);
          a[n * i + k].re -= p.re;
          a[n * i + k].im -= p.im;
        }
      }
      __syncwarp();
    }
    if (lane == 0) {
      dc r;
      if (singular) {
        r = dc{nan(""), nan("")};  // an all-zero row: flagged to the host
      } else if (!log_det) {
        r = dc{d, 0.0};
        for (int i = 0; i < n; ++i) r = dmul(r, a[n * i + i]);
      } else {
        r = dc{log(fabs(d)), d < 0 ? 3.14159265358979323846 : 0.0};
        for (int i = 0; i < n; ++i) {
          r.re += log(dabs(a[n * i + i]));
          r.im += atan2(a[n * i + i].im, a[n * i + i].re);
        }
      }
      double* o = out + c * out_conf_stride + out_offset + 2L * m;
      o[0] = r.re;
      o[1] = r.im;
    }
    __syncwarp();
  }
}

// N <= 32: a segment of a warp per (matrix, measured minor) -- 8 lanes for
// minors up to 8, 16 up to 16, the warp above -- lane i holding row i in
// registers.  The elimination of slater_dets_warp_kernel; rows stay in their
// lanes and carry their position instead of being swapped.  Column j is always
// a[0]: a step's update writes entry k + 1 into place k, so the loop over j is
// not unrolled and the code stays small (unrolled it would not fit the
// instruction cache, with warps at different steps).  The pivot row and its
// pivot's reciprocal (every row forms its own, beside the search) go through
// shared memory.  Pivots are compared by |a|^2 / max|row|^2 -- the order of
// |a| / max|row|, exact ties to the last position as before -- so that no
// hypot is taken; where a square under- or overflows the moduli themselves are
// compared.
//
// Bound by the latency of a step (search, reciprocal, broadcast) at 16 warps
// per SM and by instruction issue (half of the cycles): 4096 matrices of N = 19
// take 191 us (a warp per minor in shared memory: 504; a warp per minor in
// registers, no segments: 319), 4096 of N = 7 with struck columns 30 (130), 500 of
// N = 32 161 (346).
constexpr int kRowLuWarps = 4;
constexpr int kRowLuMax = 32;

__device__ __forceinline__ double dnorm2(dc a) { return fma(a.re, a.re, a.im * a.im); }

// The largest of v over the SEG lanes of a segment
template <int SEG>
__device__ __forceinline__ unsigned seg_max(unsigned v) {
  if constexpr (SEG == 32) {
    return __reduce_max_sync(0xffffffffu, v);
  } else {
#pragma unroll
    for (int off = SEG / 2; off > 0; off >>= 1) v = max(v, __shfl_xor_sync(0xffffffffu, v, off));
    return v;
  }
}

// The minor of order n of configuration c (measured minor m), by the SEG lanes
// of a segment; n = 0: none (a segment past the last minor).  Every segment of
// a warp goes through the steps of the largest minor in it.  urow: the
// segment's two pivot rows.
template <int SEG, int NMAX, int MODE>
__device__ __forceinline__ void minor_lu(const double2* __restrict__ S, const double2* __restrict__ psi1, int N,
                                         long c, int m, int n, int log_det, double* __restrict__ out,
                                         double2 (*urow)[NMAX + 1]) {
  static_assert(NMAX % 4 == 0 && NMAX <= SEG, "rows live in lanes, columns in groups of four");
  constexpr double kTiny = 1e-280, kHuge = 1e280;
  const unsigned all = 0xffffffffu;
  const int lane = threadIdx.x & (SEG - 1), first = (threadIdx.x & 31) & ~(SEG - 1);
  const unsigned seg_mask = (SEG == 32 ? all : (1u << (SEG & 31)) - 1u) << first;
  const int steps = SEG == 32 ? n : (int)__reduce_max_sync(all, (unsigned)n);
  const int at = lane < n ? lane : 0;  // (lanes past the minor hold a copy of its first row, unused)
  const double2* row = S + (c * N + at) * N;
  dc a[NMAX];
#pragma unroll
  for (int k = 0; k < NMAX; ++k) a[k] = dc{0.0, 0.0};
#pragma unroll
  for (int k4 = 0; k4 < NMAX; k4 += 4) {
    if (k4 >= steps) break;
#pragma unroll
    for (int k = k4; k < k4 + 4; ++k)
      if (k < n) {
        // SlaterDet2::Run column n - 1 from psi1[s + (n - 1) N] (slater_det2.C:102-106)
        const double2* from = MODE && m % 2 == 0 && k == n - 1 ? psi1 + (c * N + n - 1) * N + at : row + k;
        const double2 v = *from;
        a[k] = dc{v.x, v.y};
      }
  }
  double big = 0.0;  // the row's largest |a|^2
#pragma unroll
  for (int k = 0; k < NMAX; ++k) big = fmax(big, dnorm2(a[k]));
  bool zero_row = lane < n && big == 0.0;
  const bool plain = !(__ballot_sync(all, lane < n && !(big > kTiny && big < kHuge)) & seg_mask);
  double inv_big = 1.0 / big;  // 1 / max|row|^2, or 1 / max|row| by moduli
  if (!plain) {
    big = 0.0;
#pragma unroll
    for (int k = 0; k < NMAX; ++k) big = fmax(big, dabs(a[k]));
    zero_row = lane < n && big == 0.0;
    inv_big = 1.0 / big;
  }
  const bool singular = __ballot_sync(all, zero_row) & seg_mask;
  double d = 1.0;
  dc mine{1.0, 0.0};  // the pivot of step `lane`
  int pos = lane;     // this row's position after the swaps so far
  for (int j = 0; j < steps; ++j) {
    const int rem = steps - j;
    const bool live = lane < n && pos >= j && j < n;
    // the pivot this row would be, and its reciprocal
    const bool zero = a[0].re == 0.0 && a[0].im == 0.0;
    const dc z = zero ? dc{1.0e-20, 0.0} : a[0];
    const double q = dnorm2(z);
    double key = live && !zero ? (plain ? q : dabs(z)) * inv_big : 0.0;
    unsigned hi = (unsigned)__double2hiint(key);
    unsigned mhi = seg_max<SEG>(hi);
    dc r;
    {
      const double inv = 1.0 / q;
      r = dc{z.re * inv, -z.im * inv};
      if (!(q > kTiny && q < kHuge)) r = drecip(z);
    }
    if (__any_sync(all, plain && j < n && mhi < 0x05000000u)) {
      // every square of a segment below 1e-284 of its row's: compare its moduli
      const bool low = plain && mhi < 0x05000000u;
      if (low) key = live && !zero ? dabs(z) * sqrt(inv_big) : 0.0;
      hi = (unsigned)__double2hiint(key);
      mhi = seg_max<SEG>(hi);
    }
    unsigned cand = __ballot_sync(all, live && hi == mhi) & seg_mask;
    if (__any_sync(all, cand & (cand - 1))) {  // more than one: the keys' lower halves, then the last position
      const unsigned lo = (unsigned)__double2loint(key);
      const bool in = live && hi == mhi;
      const unsigned mlo = seg_max<SEG>(in ? lo : 0u);
      const unsigned last = seg_max<SEG>(in && lo == mlo ? (unsigned)pos + 1u : 0u);
      cand = __ballot_sync(all, in && lo == mlo && (unsigned)pos + 1u == last) & seg_mask;
    }
    const int at_lane = cand ? __ffs(cand) - 1 : first;
    const bool pivot = live && (int)(threadIdx.x & 31) == at_lane;
    double2* u = urow[j & 1];
    if (pivot) {
      u[NMAX] = make_double2(r.re, r.im);
      u[0] = make_double2(z.re, z.im);
#pragma unroll
      for (int k4 = 0; k4 < NMAX; k4 += 4) {
        if (k4 >= rem) break;
#pragma unroll
        for (int k = k4; k < k4 + 4; ++k)
          if (k > 0) u[k] = make_double2(a[k].re, a[k].im);
      }
    }
    const int imax = __shfl_sync(all, pos, at_lane);
    if (imax != j) {
      if (j < n) d = -d;
      if (live && pos == j) pos = imax;  // (the pivot row takes position j)
    }
    if (pivot) pos = j;
    __syncwarp();
    if (lane == j && j < n) mine = dc{u[0].x, u[0].y};
    const dc l = dmul(a[0], dc{u[NMAX].x, u[NMAX].y});  // (rows above are eliminated too, unread)
#pragma unroll
    for (int k4 = 0; k4 < NMAX; k4 += 4) {
      if (k4 + 1 >= rem) break;
#pragma unroll
      for (int k = k4; k < k4 + 4; ++k) {
        if (k + 1 < NMAX) {
          const double2 w = u[k + 1];
          // the product by itself, then one rounding at the entry's size: nested
          // FMAs round there twice, 3 % less time and 1.4 times the error (rms over
          // matrices 1 + 0.3 G of N = 19: 0.57e-15 against 0.41e-15, as before)
          const dc p{fma(l.re, w.x, -(l.im * w.y)), fma(l.re, w.y, l.im * w.x)};
          a[k] = dc{a[k + 1].re - p.re, a[k + 1].im - p.im};
        }
      }
    }
  }
  // the product (or the sum of logs) of the pivots
  dc v = mine;
  if (log_det) v = lane < n ? dc{log(dabs(mine)), atan2(mine.im, mine.re)} : dc{0.0, 0.0};
#pragma unroll
  for (int off = SEG / 2; off > 0; off >>= 1) {
    const dc w{__shfl_xor_sync(all, v.re, off), __shfl_xor_sync(all, v.im, off)};
    v = log_det ? dc{v.re + w.re, v.im + w.im} : dmul(v, w);
  }
  if (lane == 0 && n > 0) {
    if (singular) v = dc{nan(""), nan("")};  // an all-zero row: flagged to the host
    else if (log_det) v.im += d < 0 ? 3.14159265358979323846 : 0.0;
    else v = dc{d * v.re, d * v.im};
    out[2L * m] = v.re;
    out[2L * m + 1] = v.im;
  }
  __syncwarp();  // the pivot rows have been read
}

// Minors of orders lo + 1 .. hi of every configuration, SEG lanes each, by the
// blocks b0, b0 + 1, .. of a launch
template <int SEG, int NMAX, int MODE>
__device__ __forceinline__ void minor_class(const double2* S, const double2* psi1, int N, int nconf, int lo, int hi,
                                            int log_det, double* out, long out_conf_stride, long block,
                                            double2* smem) {
  constexpr int PER = 32 / SEG;
  const int warp = threadIdx.x >> 5, seg = (threadIdx.x & 31) / SEG;
  const int per_conf = (MODE ? 2 : 1) * (hi - lo);
  const long g = (block * kRowLuWarps + warp) * PER + seg;
  long c = g / per_conf;
  int m = (MODE ? 2 * lo : lo) + (int)(g - c * per_conf);
  int n = (MODE ? m / 2 : m) + 1;
  if (c >= nconf) c = nconf - 1, n = 0;
  minor_lu<SEG, NMAX, MODE>(S, psi1, N, c, m, n, log_det, out + c * out_conf_stride,
                            reinterpret_cast<double2(*)[NMAX + 1]>(smem + (warp * PER + seg) * 2 * (NMAX + 1)));
}

__host__ __device__ inline long minor_blocks(int nconf, int mode, int lo, int hi, int per) {
  const long segs = (long)nconf * (mode ? 2 : 1) * (hi > lo ? hi - lo : 0), w = (segs + per - 1) / per;
  return (w + kRowLuWarps - 1) / kRowLuWarps;
}

// NMAX: N rounded up to a multiple of four; the first blocks take the largest minors
template <int NMAX, int MODE>
__global__ void __launch_bounds__(32 * kRowLuWarps, NMAX <= 8 ? 5 : NMAX <= 20 ? 4 : 2)
    slater_dets_row_kernel(const double2* __restrict__ S, const double2* __restrict__ psi1, int N, int nconf,
                           int log_det, double* __restrict__ out, long out_conf_stride) {
  // one segment of 32 (NMAX + 1) or two of 16 or four of 8 (9) entries per warp, two rows each
  __shared__ double2 smem[kRowLuWarps * 2 * (NMAX + 1 > 36 ? NMAX + 1 : 36)];
  long b = blockIdx.x;
  if constexpr (NMAX > 16) {
    const long nb = minor_blocks(nconf, MODE, 16, N, 1);
    if (b < nb) {
      minor_class<32, NMAX, MODE>(S, psi1, N, nconf, 16, N, log_det, out, out_conf_stride, b, smem);
      return;
    }
    b -= nb;
  }
  if constexpr (NMAX > 8) {
    const int hi = N < 16 ? N : 16;
    const long nb = minor_blocks(nconf, MODE, 8, hi, 2);
    if (b < nb) {
      minor_class<16, NMAX < 16 ? NMAX : 16, MODE>(S, psi1, N, nconf, 8, hi, log_det, out, out_conf_stride, b, smem);
      return;
    }
    b -= nb;
  }
  minor_class<8, NMAX < 8 ? NMAX : 8, MODE>(S, psi1, N, nconf, 0, N < 8 ? N : 8, log_det, out, out_conf_stride, b,
                                            smem);
}

constexpr int kWarpLuMaxN = 64;
constexpr size_t kWarpLuSmemCap = 200 * 1024;

static size_t warp_lu_bytes(int N) { return (size_t)N * N * sizeof(dc) + N * sizeof(double); }
static int warp_lu_warps(int N) {
  int w = (int)(kWarpLuSmemCap / warp_lu_bytes(N));
  return w < 1 ? 1 : (w > kWarpLuMaxWarps ? kWarpLuMaxWarps : w);
}

// Leading-minor determinants by a warp per minor (N <= 64, no scratch): rows in
// registers up to N = 32 (read 16 bytes at a time: matrices that start on 16),
// the minor in shared memory otherwise.
nrcps_status slater_dets_warp(nrcps_context* ctx, const double* S, const double* psi1, int N, int nconf, int mode,
                              int log_det, double* out, long out_conf_stride, long out_offset) {
  const int nmeas = mode ? 2 * N : N;
  const long total = (long)nconf * nmeas;
  if (total == 0) return NRCPS_OK;
  if (N <= kRowLuMax && ((reinterpret_cast<uintptr_t>(S) | reinterpret_cast<uintptr_t>(psi1)) & 15) == 0) {
    const long blocks = minor_blocks(nconf, mode, 16, N, 1) + minor_blocks(nconf, mode, 8, N < 16 ? N : 16, 2) +
                        minor_blocks(nconf, mode, 0, N < 8 ? N : 8, 4);
    auto launch = [&](auto kern) {
      kern<<<(unsigned)blocks, 32 * kRowLuWarps, 0, ctx->stream>>>(
          reinterpret_cast<const double2*>(S), reinterpret_cast<const double2*>(psi1), N, nconf, log_det,
          out + out_offset, out_conf_stride);
    };
#define NRCPS_CASE(M) \
  if (N <= M) {       \
    if (mode) launch(slater_dets_row_kernel<M, 1>); \
    else launch(slater_dets_row_kernel<M, 0>);      \
  }
    NRCPS_CASE(4) else NRCPS_CASE(8) else NRCPS_CASE(12) else NRCPS_CASE(16) else NRCPS_CASE(20) else NRCPS_CASE(24)
    else NRCPS_CASE(32)
#undef NRCPS_CASE
    ctx->launches++;
    return check_launch(ctx, "slater_dets_row_kernel");
  }
  static bool attr_set[16] = {false};
  if (!attr_set[ctx->device & 15]) {
    NRCPS_TRY(check_cuda(ctx,
                         cudaFuncSetAttribute(slater_dets_warp_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                              (int)kWarpLuSmemCap),
                         "slater_dets_warp: smem attribute"));
    attr_set[ctx->device & 15] = true;
  }
  const int wpb = warp_lu_warps(N);
  const long blocks = (total + wpb - 1) / wpb;
  const unsigned g = (unsigned)(blocks < (long)ctx->sm_count * 64 ? blocks : (long)ctx->sm_count * 64);
  slater_dets_warp_kernel<<<g, 32 * wpb, (size_t)wpb * warp_lu_bytes(N), ctx->stream>>>(S, psi1, N, nconf, mode, log_det,
                                                                                   out, out_conf_stride, out_offset);
  ctx->launches++;
  return check_launch(ctx, "slater_dets_warp_kernel");
}

size_t slater_dets_scratch_bytes(int N, int nconf, int mode) {
  const int nmeas = mode ? 2 * N : N;
  return sizeof(double) * (size_t)nconf * nmeas * (2L * N * N + N);
}

// scr: caller-owned scratch of slater_dets_scratch_bytes(), or NULL for the
// context's scratch.
nrcps_status slater_dets_impl(nrcps_context* ctx, const double* S, const double* psi1, int N, int nconf, int mode,
                              int log_det, double* out, long out_conf_stride, long out_offset, double* scr) {
  const int nmeas = mode ? 2 * N : N;
  const long total = (long)nconf * nmeas;
  if (total == 0) return NRCPS_OK;
  if (!scr) {
    nrcps_status st;
    scr = (double*)scratch(ctx, slater_dets_scratch_bytes(N, nconf, mode), &st);
    if (!scr) return st;
  }
  slater_dets_kernel<<<grid_for(total, 64, 1L << 20), 64, 0, ctx->stream>>>(S, psi1, N, nconf, mode, log_det, out,
                                                                             scr, out_conf_stride, out_offset);
  ctx->launches++;
  return check_launch(ctx, "slater_dets_kernel");
}

// The determinant path of the library: the warp kernel for N <= 64 (unless
// the "lu.warp" option is 0), else the per-thread kernel with scratch.
nrcps_status slater_dets_dispatch(nrcps_context* ctx, const double* S, const double* psi1, int N, int nconf, int mode,
                                  int log_det, double* out, long out_conf_stride, long out_offset, double* scr) {
  if (N <= kWarpLuMaxN && ctx->lu_warp)
    return slater_dets_warp(ctx, S, psi1, N, nconf, mode, log_det, out, out_conf_stride, out_offset);
  return slater_dets_impl(ctx, S, psi1, N, nconf, mode, log_det, out, out_conf_stride, out_offset, scr);
}

// The chunks' sums of overlap_tile_kernel, where a second kernel adds them up:
// an ensemble, whose graph holds the address, brings a buffer of its own; a
// direct call takes the context's, of fixed size and made at the first use,
// after an event that the last call which used it recorded behind its second
// kernel -- the context's stream may be another one by now.  A call inside a
// capture takes neither: the graph may run beside later calls.
constexpr size_t kOverlapPartBytes = 32u << 20;  // (N = 19 at L = 48: 26 configurations)

static double* overlap_context_part(nrcps_context* ctx) {
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  cudaError_t e = cudaStreamIsCapturing(ctx->stream, &cs);
  if (e == cudaSuccess && cs != cudaStreamCaptureStatusNone) return nullptr;
  BesideCaptures beside;
  if (e == cudaSuccess && !ctx->overlap_done)
    e = cudaEventCreateWithFlags(&ctx->overlap_done, cudaEventDisableTiming);
  if (e == cudaSuccess && !ctx->overlap_part) e = cudaMalloc(&ctx->overlap_part, kOverlapPartBytes);
  if (e == cudaSuccess) e = cudaStreamWaitEvent(ctx->stream, ctx->overlap_done, 0);
  if (e == cudaSuccess) return (double*)ctx->overlap_part;
  cudaGetLastError();
  return nullptr;
}

// CTAs for a configuration and tile: about four per SM in all.  One takes it
// alone, a cluster has one per group; where more than four are wanted they leave
// their chunks' sums in a buffer for a second kernel (`each`): clusters of seven
// or eight do not fill the chip.  FP64, 40 configurations of N = 19, L = 32: 355 us
// against 455 by clusters, L = 24 148 against 221; 100 of them 355 and 419.
struct OvSplit {
  int ctas, per_cta;
  bool each;
};
static OvSplit overlap_split(const nrcps_context* ctx, const OvTile& o, const OvChunks& ch, int ns, int nt, int nconf,
                             bool buffer) {
  const long tiles = (long)nconf * o.ns_t * o.nt_t;
  const long want = (4L * ctx->sm_count + tiles - 1) / tiles;
  if (want <= 1 || ch.groups == 1) return {1, ch.chunks, false};
  const bool room = sizeof(double2) * (size_t)nconf * ns * nt * ch.chunks <= kOverlapPartBytes;
  if (want <= 4 || ch.chunks <= OV_GROUPS || !room || !buffer)
    return {ch.groups, ch.per_group, false};
  const long per = (ch.chunks + want - 1) / want;
  return {(int)((ch.chunks + per - 1) / per), (int)per, true};
}

static long overlap_direct_ctas(int ns, int nt, int nconf, const OvTile& o, const OvChunks& ch) {
  const long here = OD_WARPS / ch.groups * (32 / o.lanes), sb = overlap_direct_sources(ns);
  return ((long)nconf * nt + here - 1) / here * ((ns + sb - 1) / sb);
}

// Groups of five or six sources, many CTAs: three per SM, two sites in flight (N = 5,
// L = 12, 1500 configurations 113 us against 128 with two CTAs and four sites, N = 10,
// L = 16, one 17 against 12).
static bool overlap_direct_many(const nrcps_context* ctx, int ns, int nt, int nconf, const OvTile& o,
                                const OvChunks& ch) {
  const int sb = overlap_direct_sources(ns);
  return (sb == 5 || sb == 6) && overlap_direct_ctas(ns, nt, nconf, o, ch) >= 8L * ctx->sm_count;
}

// Whether the kernel without staging is the faster one, by what either takes in
// microseconds beyond a launch.  It: rounds of CTAs times the sites of a lane, and
// the loads and FMAs of every orbital with every group of sources; by tiles:
// rounds times sites of a lane, the rows staged, CTAs, and the second kernel.
// Fitted to both kernels over N = 1 .. 33, L = 8 .. 48, one to 4096 configurations
// (1324 calls): the choice costs 1 % in the mean of what always taking the faster
// one would.  In small volumes the sources stay in L1 while there are few orbitals;
// eight accumulators in large batches there, and FP32 orbitals in large batches
// elsewhere, take longer than the sum says.
// What is left against a block per orbital of 256 threads, the kernel before: N = 7, 8
// and 13 in batches of 10^5 to 10^6 sites, and one orbital of 4096 configurations, by
// up to a third (N = 7, L = 12, 512 configurations 75 against 64 us).
static bool overlap_direct_pays(const nrcps_context* ctx, int ns, int nt, int nconf, long vol, bool fp64, const OvTile& o,
                                const OvChunks& ch, const OvSplit& split) {
  const int sb = overlap_direct_sources(ns);
  const double entries = (double)nconf * nt * vol;
  const double slots = (sb <= 4 || overlap_direct_many(ctx, ns, nt, nconf, o, ch) ? 3.0 : 2.0) * ctx->sm_count;
  double direct = 0.03 * ceil(overlap_direct_ctas(ns, nt, nconf, o, ch) / slots) * ch.per_group * ch.sites / o.lanes * (sb + 1) +
                  1e-6 * entries * (0.2 * ns + 1.3 * ((ns + sb - 1) / sb));
  if (vol <= 4096 && entries < 5e6) direct *= 0.85;
  else if (vol <= 4096 && sb >= 7 && o.lanes < 32 && fp64) direct *= 1.15;
  else if (vol > 4096 && entries >= 2e7 && !fp64) direct *= 1.6;
  const double ctas = (double)nconf * o.ns_t * o.nt_t * split.ctas, sites = (double)split.per_cta * ch.sites;
  const double tiles = 1.0 + (split.each ? 3.7 : 0.0) + 0.2 * ceil(ctas / (2.0 * ctx->sm_count)) * sites / o.lanes +
                       3e-6 * ctas * sites * o.rows + 5e-3 * ctas;
  return direct < tiles;
}

// What an ensemble of these overlaps brings for the sums (0: nothing).
size_t overlap_part_bytes(nrcps_context* ctx, int ns, int nt, int nconf, long vol, nrcps_precision prec) {
  OvTile o = overlap_tiles(ns, nt);
  const OvChunks ch = overlap_chunks(vol, o);
  const OvSplit split = overlap_split(ctx, o, ch, ns, nt, nconf, true);
  if (!split.each || overlap_direct_pays(ctx, ns, nt, nconf, vol, prec == NRCPS_F64, o, ch, split)) return 0;
  return sizeof(double2) * (size_t)nconf * ns * nt * ch.chunks;
}

template <typename R>
static nrcps_status launch_overlap(nrcps_context* ctx, const double* src, int ns, const void* psi, int nt, int nconf,
                                   long vol, double* S, double* part) {
  OvTile o = overlap_tiles(ns, nt);
  const OvChunks ch = overlap_chunks(vol, o);
  OvSplit split = overlap_split(ctx, o, ch, ns, nt, nconf, true);
  if (overlap_direct_pays(ctx, ns, nt, nconf, vol, sizeof(R) == 8, o, ch, split)) {
    const long orbitals = (long)nconf * nt, here = OD_WARPS / ch.groups * (32 / o.lanes);
    const int sb = overlap_direct_sources(ns);
    auto launch = [&](auto kern) {
      kern<<<dim3((unsigned)((orbitals + here - 1) / here), (unsigned)((ns + sb - 1) / sb)), 32 * OD_WARPS, 0,
             ctx->stream>>>(reinterpret_cast<const double2*>(src), ns, psi, nt, vol, orbitals, ch, S);
    };
    const bool many = overlap_direct_many(ctx, ns, nt, nconf, o, ch);
    auto lanes = [&](auto l) {
      constexpr int LANES = decltype(l)::value;
      switch (2 * sb + many) {
        case 4: return launch(overlap_direct_kernel<R, 2, LANES, false>);
        case 8: return launch(overlap_direct_kernel<R, 4, LANES, false>);
        case 10: return launch(overlap_direct_kernel<R, 5, LANES, false>);
        case 11: return launch(overlap_direct_kernel<R, 5, LANES, true>);
        case 12: return launch(overlap_direct_kernel<R, 6, LANES, false>);
        case 13: return launch(overlap_direct_kernel<R, 6, LANES, true>);
        case 14: return launch(overlap_direct_kernel<R, 7, LANES, false>);
        default: return launch(overlap_direct_kernel<R, 8, LANES, false>);
      }
    };
    if (o.lanes == 8) lanes(std::integral_constant<int, 8>());
    else if (o.lanes == 16) lanes(std::integral_constant<int, 16>());
    else lanes(std::integral_constant<int, 32>());
    ctx->launches++;
    return check_launch(ctx, "overlap_direct_kernel");
  }
  const size_t smem = sizeof(double2) * (2 * (size_t)o.rows * o.T + 2 * 16 * o.ts * o.tt);
  // (132 rows of 32 sites and 32 blocks are the most)
  NRCPS_TRY(allow_smem(ctx, (const void*)overlap_tile_kernel<R>, 160 * 1024, "overlap_tile: smem attribute"));
  bool shared = false;
  if (split.each && !part) {
    part = overlap_context_part(ctx);
    shared = part != nullptr;
    if (!part) split = overlap_split(ctx, o, ch, ns, nt, nconf, false);
  }
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = split.each ? 1u : (unsigned)split.ctas;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.gridDim = dim3((unsigned)((long)nconf * o.ns_t * o.nt_t * split.ctas));
  cfg.blockDim = dim3(OV_THREADS);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = ctx->stream;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  ctx->launches++;
  NRCPS_TRY(check_cuda(ctx, cudaLaunchKernelEx(&cfg, overlap_tile_kernel<R>, reinterpret_cast<const double2*>(src), ns,
                                               psi, nt, nconf, vol, split.ctas, split.per_cta, split.each ? 1 : 0, ch,
                                               o, split.each ? part : S),
                       "overlap_tile_kernel launch"));
  if (split.each) {
    const long per_conf = (long)ns * nt, total = nconf * per_conf;
    overlap_sum_kernel<<<grid_for(total, 64), 64, 0, ctx->stream>>>(reinterpret_cast<const double2*>(part), ch,
                                                                    per_conf, total, S);
    ctx->launches++;
    const nrcps_status st = check_launch(ctx, "overlap_sum_kernel");
    if (shared)
      NRCPS_TRY(check_cuda(ctx, cudaEventRecord(ctx->overlap_done, ctx->stream), "overlap: event record"));
    return st;
  }
  return NRCPS_OK;
}

// part: the caller's buffer of overlap_part_bytes() for the chunks' sums, or
// null for the context's.
nrcps_status overlap_impl(nrcps_context* ctx, const double* src, int ns, const void* psi, int nt, int nconf,
                          long vol, nrcps_precision prec, double* S, double* part) {
  if ((long)nconf * nt * ns == 0) return NRCPS_OK;
  return prec == NRCPS_F64 ? launch_overlap<double>(ctx, src, ns, psi, nt, nconf, vol, S, part)
                           : launch_overlap<float>(ctx, src, ns, psi, nt, nconf, vol, S, part);
}

nrcps_status gather_impl(nrcps_context* ctx, const int* index, int ns, const void* psi, int nt, int nconf, long vol,
                         nrcps_precision prec, double* S) {
  long total = (long)nconf * ns * nt;
  if (total == 0) return NRCPS_OK;
  unsigned g = grid_for(total, 256, (long)ctx->sm_count * 8);
  if (prec == NRCPS_F64) gather_kernel<double><<<g, 256, 0, ctx->stream>>>(index, ns, psi, nt, nconf, vol, S);
  else gather_kernel<float><<<g, 256, 0, ctx->stream>>>(index, ns, psi, nt, nconf, vol, S);
  ctx->launches++;
  return check_launch(ctx, "gather_kernel");
}

template <typename R>
static nrcps_status launch_pair_tile(nrcps_context* ctx, const void* psi1, const void* psi2, int n, int nconf,
                                     long vol, const double* w, const int* opp, const int* flags, int host_flags,
                                     bool leave_sym, double* phi) {
  using Sh = PairShape<R>;
  const int ts = Sh::ts(n);
  const size_t smem = Sh::smem(n);
  static bool attr_set[16] = {false};
  if (!attr_set[ctx->device & 15]) {
    size_t most = 0;
    for (int m = 1; m <= PAIR_MAXN; ++m) most = Sh::smem(m) > most ? Sh::smem(m) : most;
    NRCPS_TRY(check_cuda(ctx, cudaFuncSetAttribute(pair_tile_kernel<R>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                   (int)most),
                         "pair_tile: smem attribute"));
    attr_set[ctx->device & 15] = true;
  }
  // CTAs per configuration: enough CTAs for about four per SM, at most 8
  // (a portable cluster) and no more than the tiles
  const long ntiles = (vol + ts - 1) / ts;
  int split = (int)((4L * ctx->sm_count + nconf - 1) / nconf);
  if (split > 8) split = 8;
  if (split > ntiles) split = (int)ntiles;
  if (split < 1) split = 1;
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)split;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.gridDim = dim3((unsigned)((long)nconf * split));
  cfg.blockDim = dim3(PAIR_THREADS);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = ctx->stream;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cudaError_t e =
      cudaLaunchKernelEx(&cfg, pair_tile_kernel<R>, psi1, psi2, n, vol, w, opp, flags, host_flags, leave_sym ? 1 : 0,
                         ts, phi);
  ctx->launches++;
  return check_cuda(ctx, e, "pair_tile_kernel launch");
}

bool pair_sym_supported(int n, long vol);  // pair_sym.cu
nrcps_status pair_sym(nrcps_context* ctx, const void* psi, int n, int nconf, long vol, const double* w, const int* opp,
                      const int* flags, double* phi);

// props: the table's properties as the caller checked them on the host
// (pair_table_props), or -1: the device checks them before the tiles.
nrcps_status pair_impl(nrcps_context* ctx, const void* psi1, const void* psi2, int n, int nconf, long vol,
                       const double* w, const int* opp, nrcps_precision prec, double* phi, int props) {
  long blocks = (long)nconf * n * n;
  if (blocks == 0) return NRCPS_OK;
  if (n <= PAIR_MAXN && ctx->pair_tile && (long)nconf * 8 < (1L << 31)) {
    const int* flags = nullptr;
    if (props < 0) {
      NRCPS_TRY(check_cuda(ctx, cudaMemsetAsync(ctx->dev_pair_flag, 0, sizeof(int), ctx->stream), "pair flag"));
      opp_involution_check_kernel<<<grid_for(vol, 256), 256, 0, ctx->stream>>>(opp, w, vol, ctx->dev_pair_flag);
      ctx->launches++;
      NRCPS_TRY(check_launch(ctx, "opp_involution_check_kernel"));
      flags = ctx->dev_pair_flag;
    }
    if (prec == NRCPS_F64)
      return launch_pair_tile<double>(ctx, psi1, psi2, n, nconf, vol, w, opp, flags, props, false, phi);
    // one set of FP32 orbitals: the packed kernel where the table qualifies;
    // a table checked on the device decides there which of the two runs
    const bool one_set = psi1 == psi2 && pair_sym_supported(n, vol);
    if (one_set && (flags || !props)) {
      NRCPS_TRY(pair_sym(ctx, psi1, n, nconf, vol, w, opp, flags, phi));
      if (!flags) return NRCPS_OK;
    }
    return launch_pair_tile<float>(ctx, psi1, psi2, n, nconf, vol, w, opp, flags, props, one_set && flags, phi);
  }
  if (prec == NRCPS_F64) pair_kernel<double><<<(unsigned)blocks, 256, 0, ctx->stream>>>(psi1, psi2, n, vol, w, opp, phi);
  else pair_kernel<float><<<(unsigned)blocks, 256, 0, ctx->stream>>>(psi1, psi2, n, vol, w, opp, phi);
  ctx->launches++;
  return check_launch(ctx, "pair_kernel");
}

}  // namespace nrcps

using namespace nrcps;

extern "C" nrcps_status nrcps_overlap(nrcps_context* ctx, const double* dev_src, int ns, const void* dev_psi, int nt,
                                      int nconf, long vol, nrcps_precision prec, double* dev_S) {
  if (!ctx) return NRCPS_ERR_INVALID_ARGUMENT;
  NRCPS_REQUIRE(ctx, ns >= 0 && nt >= 0 && nconf >= 0 && vol > 0, "nrcps_overlap: bad arguments");
  if ((long)ns * nt * nconf == 0) return NRCPS_OK;  // empty batch: nothing to read or write
  NRCPS_REQUIRE(ctx, dev_src && dev_psi && dev_S, "nrcps_overlap: null pointer");
  if (prec == NRCPS_F32 && ctx->overlap_tc && ns > 0 && nt > 0 && nconf > 0 && ((uintptr_t)dev_psi & 15) == 0 &&
      overlap_tc_supported(vol, ns, nt, nconf)) {
    const size_t need = overlap_tc_split_bytes(ns, vol);
    if (need > ctx->tc_split_bytes) {
      if (ctx->tc_split) {
        cudaStreamSynchronize(ctx->stream);
        cudaFree(ctx->tc_split);
        ctx->tc_split = nullptr;
        ctx->tc_split_bytes = 0;
      }
      NRCPS_TRY(check_cuda(ctx, cudaMalloc(&ctx->tc_split, need), "cudaMalloc(overlap split)"));
      ctx->tc_split_bytes = need;
    }
    NRCPS_TRY(overlap_tc_prepare(ctx, dev_src, ns, vol, nt, nconf, (float*)ctx->tc_split));
    return overlap_tc(ctx, (const float*)ctx->tc_split, ns, dev_psi, nt, nconf, vol, dev_S);
  }
  return overlap_impl(ctx, dev_src, ns, dev_psi, nt, nconf, vol, prec, dev_S, nullptr);
}

extern "C" nrcps_status nrcps_overlap_planewave(nrcps_context* ctx, const int* dev_index, int ns, const void* dev_psi,
                                                int nt, int nconf, long vol, nrcps_precision prec, double* dev_S) {
  if (!ctx) return NRCPS_ERR_INVALID_ARGUMENT;
  NRCPS_REQUIRE(ctx, ns >= 0 && nt >= 0 && nconf >= 0 && vol > 0, "nrcps_overlap_planewave: bad arguments");
  if ((long)ns * nt * nconf == 0) return NRCPS_OK;
  NRCPS_REQUIRE(ctx, dev_index && dev_psi && dev_S, "nrcps_overlap_planewave: null pointer");
  return gather_impl(ctx, dev_index, ns, dev_psi, nt, nconf, vol, prec, dev_S);
}

extern "C" nrcps_status nrcps_pair_matrix(nrcps_context* ctx, const void* dev_psi1, const void* dev_psi2, int n,
                                          int nconf, long vol, const double* dev_w, const int* dev_opposite,
                                          nrcps_precision prec, double* dev_phi) {
  if (!ctx) return NRCPS_ERR_INVALID_ARGUMENT;
  NRCPS_REQUIRE(ctx, n >= 0 && nconf >= 0 && vol > 0, "nrcps_pair_matrix: bad arguments");
  if ((long)n * nconf == 0) return NRCPS_OK;
  NRCPS_REQUIRE(ctx, dev_psi1 && dev_psi2 && dev_w && dev_opposite && dev_phi, "nrcps_pair_matrix: null pointer");
  return pair_impl(ctx, dev_psi1, dev_psi2, n, nconf, vol, dev_w, dev_opposite, prec, dev_phi, -1);
}

extern "C" nrcps_status nrcps_shifted_pair_matrix(nrcps_context* ctx, const void* dev_psi1, const void* dev_psi2,
                                                  int n, int nconf, long vol, int nterms, const int* dev_shift,
                                                  const double* dev_wl, const int* dev_opposite,
                                                  nrcps_precision prec, double* dev_phi) {
  if (!ctx) return NRCPS_ERR_INVALID_ARGUMENT;
  NRCPS_REQUIRE(ctx, n >= 0 && nconf >= 0 && vol > 0 && nterms > 0, "nrcps_shifted_pair_matrix: bad arguments");
  const long blocks = (long)nconf * n * n;
  if (blocks == 0) return NRCPS_OK;
  NRCPS_REQUIRE(ctx, dev_psi1 && dev_psi2 && dev_shift && dev_wl && dev_opposite && dev_phi,
                "nrcps_shifted_pair_matrix: null pointer");
  if (prec == NRCPS_F64)
    shifted_pair_kernel<double><<<(unsigned)blocks, 256, 0, ctx->stream>>>(dev_psi1, dev_psi2, n, vol, nterms,
                                                                          dev_shift, dev_wl, dev_opposite, dev_phi);
  else
    shifted_pair_kernel<float><<<(unsigned)blocks, 256, 0, ctx->stream>>>(dev_psi1, dev_psi2, n, vol, nterms,
                                                                         dev_shift, dev_wl, dev_opposite, dev_phi);
  ctx->launches++;
  return check_launch(ctx, "shifted_pair_kernel");
}

extern "C" nrcps_status nrcps_inner_product_ptrs(nrcps_context* ctx, const double* const* dev_kets,
                                                 const double* const* dev_bras, int nf, long vol, double* dev_mat) {
  if (!ctx) return NRCPS_ERR_INVALID_ARGUMENT;
  NRCPS_REQUIRE(ctx, dev_kets && dev_bras && dev_mat && nf >= 0 && vol > 0, "nrcps_inner_product_ptrs: bad arguments");
  if (nf == 0) return NRCPS_OK;
  inner_ptrs_kernel<<<(unsigned)(nf * nf), 256, 0, ctx->stream>>>(dev_kets, dev_bras, nf, vol, dev_mat);
  ctx->launches++;
  return check_launch(ctx, "inner_ptrs_kernel");
}

extern "C" nrcps_status nrcps_pair_matrix_ptrs(nrcps_context* ctx, const double* const* dev_props1,
                                               const double* const* dev_props2, int nf, long vol, const double* dev_w,
                                               const int* dev_opposite, double* dev_phi) {
  if (!ctx) return NRCPS_ERR_INVALID_ARGUMENT;
  NRCPS_REQUIRE(ctx, dev_props1 && dev_props2 && dev_w && dev_opposite && dev_phi && nf >= 0 && vol > 0,
                "nrcps_pair_matrix_ptrs: bad arguments");
  if (nf == 0) return NRCPS_OK;
  pair_ptrs_kernel<<<(unsigned)(nf * nf), 256, 0, ctx->stream>>>(dev_props1, dev_props2, nf, vol, dev_w,
                                                                 dev_opposite, dev_phi);
  ctx->launches++;
  return check_launch(ctx, "pair_ptrs_kernel");
}

extern "C" nrcps_status nrcps_slater_dets(nrcps_context* ctx, const double* dev_S, const double* dev_psi1, int N,
                                          int nconf, int mode, int log_det, double* dev_out) {
  if (!ctx) return NRCPS_ERR_INVALID_ARGUMENT;
  NRCPS_REQUIRE(ctx, N > 0 && nconf >= 0 && (mode == 0 || mode == 1), "nrcps_slater_dets: bad arguments");
  if (nconf == 0) return NRCPS_OK;
  NRCPS_REQUIRE(ctx, dev_S && dev_out && (mode == 0 || dev_psi1), "nrcps_slater_dets: null pointer");
  const int nmeas = mode ? 2 * N : N;
  return slater_dets_dispatch(ctx, dev_S, dev_psi1, N, nconf, mode, log_det, dev_out, 2L * nmeas, 0, nullptr);
}

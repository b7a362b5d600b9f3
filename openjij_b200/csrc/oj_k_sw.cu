// Swendsen-Wang cluster updates for sparse Ising graphs, one CTA per replica
// (state in shared memory up to sw_max_sites() spins, in global memory above).
//
// The reference's SwendsenWang updater (include/openjij/updater/swendsen_wang.hpp:43-182)
// works on the n spins plus the dummy spin n that carries the fields (bond
// (i, n) with coupling h_i).  One update:
//   1. every bond (i, j), i < j, that is satisfied (J s_i s_j < 0) is kept
//      with probability 1 - exp(-2 beta |J|);
//   2. the kept bonds define clusters (union-find);
//   3. every cluster flips with probability 1/2.
// Here, per replica and sweep, in shared memory:
//   1. bond e is kept when -ln(u_e) < 2 beta |J| (FP32; the same event as
//      u'_e < 1 - exp(-2 beta |J|) with u' = 1 - u), u_e from
//      Philox((e >> 2, k, r, TAG_SW_BOND))[e & 3];
//   2. union-find with lock-free hooking of the larger root under the smaller
//      one, so every cluster's root is its smallest site, whatever the order
//      in which the threads hook;
//   3. the cluster of the dummy spin stays, every other cluster flips when bit 0
//      of Philox((root >> 2, k, r, TAG_SW_FLIP))[root & 3] is set.  Holding
//      the dummy fixed leaves the distribution of the physical spins s_i s_n
//      unchanged (get_solution, include/openjij/result/get_solution.hpp:39-49,
//      reads s_i s_n): flipping the dummy's cluster with probability 1/2 is
//      the same as flipping every other cluster once more with probability 1/2.
// The partition into clusters does not depend on thread timing, so the result
// is a pure function of seed, sweep, replica and state.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "oj_device.cuh"
#include "oj_internal.h"

namespace oj {
namespace {

constexpr int kSwThreads = 512;
constexpr int kSwHookThreads = 1024;  // most threads of the hooking kernel
constexpr size_t kSwHookSmemBytes = 220 * 1024;

struct SwArgs {
  const int32_t* ei;   // [ne] bond endpoints, ei < ej (ej == n: the dummy spin)
  const int32_t* ej;
  const float* w;      // [ne] |J| of the bond (FP32)
  const uint8_t* pos;  // [ne] 1 when J > 0
  const int4* quad;    // [nq][2] four bonds: ei | ej << 16, J (FP32 bits), padded with J = 0
  int ne, n, nq;
  int8_t* spins;       // [R][n]
  const float* betas;  // [nsweeps]
  int64_t nsweeps;
  ojd::Keys keys;
  uint32_t sweep0, rep0;
};

// Parent links live in shared memory (SMEM) or, for graphs too large for it,
// in a global scratch array; there they are read past L1 (__ldcg), which does
// not see the L2 atomics of the other threads.
template <bool SMEM>
__device__ __forceinline__ uint32_t ld_parent(const uint32_t* p) {
  if constexpr (SMEM) {
    return *p;
  } else {
    return __ldcg(p);
  }
}

template <bool SMEM>
__device__ __forceinline__ uint32_t find_root(uint32_t* parent, uint32_t x) {
  uint32_t p = ld_parent<SMEM>(parent + x);
  while (p != x) {
    const uint32_t gp = ld_parent<SMEM>(parent + p);
    if (gp != p) parent[x] = gp;  // path halving (only ever points a node at an ancestor)
    x = p;
    p = gp;
  }
  return x;
}

template <bool SMEM>
__device__ __forceinline__ void unite(uint32_t* parent, uint32_t a, uint32_t b) {
  for (int guard = 0; guard < (1 << 20); ++guard) {
    a = find_root<SMEM>(parent, a);
    b = find_root<SMEM>(parent, b);
    if (a == b) return;
    if (a < b) {
      const uint32_t t = a;
      a = b;
      b = t;
    }
    // hook the larger root under the smaller; retry if a moved meanwhile
    if (atomicCAS(&parent[a], a, b) == a) return;
  }
}

// Large graphs, and calls with few replicas (sw_hooks).  What bounds sw_kernel there
// is the serial chains of its unions: lanes walk to their roots and retry at
// different lengths.  Here no lane walks: a pass hooks the larger root of every kept
// bond between two trees under the smaller with one atomic minimum, then all links
// jump to their roots together; passes go on until no kept bond joins two trees.  The
// coins are drawn four a Philox call, spins are bits, a bond is one 8-byte entry,
// and the kept test takes the hardware logarithm first (neglog_gap).  One CTA per
// replica.  Shared memory: parent[n + 1] | spin bits | coin bits | kept bonds.
// Measured (us a sweep, sw_kernel / this one): lattice 128 x 128, 16 replicas 97 / 44,
// 1024 replicas 419 / 300; lattice 64 x 64, 16 replicas 19.1 / 13.0, but 256 replicas
// 23.8 / 23.3 and 1024 replicas 65.4 / 67.3; Chimera 16 x 16 cells with fields, 16
// replicas 18.3 / 10.2, 256 replicas 22.2 / 17.9.
template <int MAXT, int MINB>
__global__ void __launch_bounds__(MAXT, MINB) sw_hook_kernel(SwArgs a) {
  extern __shared__ __align__(16) uint32_t parent[];
  __shared__ uint32_t dummy_root;
  const int n = a.n, T = blockDim.x, nw = (n + 32) >> 5;
  uint32_t* sb = parent + n + 1;
  uint32_t* coin = sb + nw;
  uint8_t* kept = reinterpret_cast<uint8_t*>(coin + nw);  // four bits per quad
  const int r = blockIdx.x, lane = threadIdx.x & 31, base = threadIdx.x - lane;
  int8_t* gs = a.spins + (size_t)r * n;
  for (int x0 = base; x0 <= n; x0 += T) {  // whole warps: x0 a multiple of 32
    const int x = x0 + lane;
    const uint32_t w = __ballot_sync(0xffffffffu, x < n && gs[x] < 0);
    if (lane == 0) sb[x0 >> 5] = w;
    if (x <= n) parent[x] = (uint32_t)x;
  }
  __syncthreads();
  const uint32_t rg = a.rep0 + (uint32_t)r;
  float bnext = a.nsweeps > 0 ? __ldg(a.betas) : 0.0f;
  for (int64_t k = 0; k < a.nsweeps; ++k) {
    const float beta2 = __fmul_rn(2.0f, bnext);
    if (k + 1 < a.nsweeps) bnext = __ldg(a.betas + k + 1);
    const uint32_t kk = a.sweep0 + (uint32_t)k;
    // 1. bonds, four per thread and Philox call; a kept bond hooks its larger
    // end under its smaller one unless that has a smaller parent already
    uint32_t low = (uint32_t)n;  // the dummy spin's smallest kept neighbour
    for (int q0 = base; q0 < a.nq; q0 += T) {
      const int q = q0 + lane;
      uint32_t nib = 0u;
      if (q < a.nq) {
        const int4 b0 = __ldg(a.quad + 2 * q), b1 = __ldg(a.quad + 2 * q + 1);
        const ojd::u4 u = ojd::philox((uint32_t)q, kk, rg, ojd::TAG_SW_BOND, a.keys);
        const uint32_t ends[4] = {(uint32_t)b0.x, (uint32_t)b0.z, (uint32_t)b1.x, (uint32_t)b1.z};
        const uint32_t js[4] = {(uint32_t)b0.y, (uint32_t)b0.w, (uint32_t)b1.y, (uint32_t)b1.w};
        bool near = false;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const uint32_t i = ends[e] & 0xFFFFu, j = ends[e] >> 16;
          // bit 0: satisfied (J s_i s_j < 0); the dummy spin is +1
          const uint32_t sat = (sb[i >> 5] >> (i & 31u)) ^ (sb[j >> 5] >> (j & 31u)) ^ (js[e] >> 31);
          const float y = __fmul_rn(beta2, __uint_as_float(js[e] & 0x7FFFFFFFu));
          const float t = ojd::neglog_gap(y, ojd::pick(u, e));  // 2 beta |J| - (-ln u)
          near = near || fabsf(t) <= ojd::kNegLogTol;
          if ((sat & 1u) && t > 0.0f) nib |= 1u << e;
        }
        if (near) {
          nib = 0u;
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const uint32_t i = ends[e] & 0xFFFFu, j = ends[e] >> 16;
            const uint32_t sat = (sb[i >> 5] >> (i & 31u)) ^ (sb[j >> 5] >> (j & 31u)) ^ (js[e] >> 31);
            if ((sat & 1u) && ojd::neglog(ojd::pick(u, e)) < __fmul_rn(beta2, __uint_as_float(js[e] & 0x7FFFFFFFu)))
              nib |= 1u << e;
          }
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const uint32_t i = ends[e] & 0xFFFFu, j = ends[e] >> 16;
          if ((nib >> e) & 1u) {
            if (j < (uint32_t)n) atomicMin(parent + j, i);
            else low = min(low, i);
          }
        }
      }
      if (q < a.nq) kept[q] = (uint8_t)nib;
    }
    low = __reduce_min_sync(0xffffffffu, low);
    if (lane == 0 && low < (uint32_t)n) atomicMin(parent + n, low);
    __syncthreads();
    // the coins of all sites, four per Philox call (a root's is read)
    for (int q0 = base; 4 * q0 < n; q0 += T) {
      const ojd::u4 c = ojd::philox((uint32_t)(q0 + lane), kk, rg, ojd::TAG_SW_FLIP, a.keys);
      uint32_t nib = ((c.x & 1u) | ((c.y & 1u) << 1) | ((c.z & 1u) << 2) | ((c.w & 1u) << 3)) << (4 * (lane & 7));
#pragma unroll
      for (int o = 1; o < 8; o <<= 1) nib |= __shfl_xor_sync(0xffffffffu, nib, o);
      if ((lane & 7) == 0 && 4 * (q0 + lane) <= n) coin[(q0 + lane) >> 3] = nib;
    }
    // 2. passes until every kept bond has both ends under one root: flatten the
    // trees (every site's link moves up to four steps a round until it is a
    // root), then every kept bond between two trees hooks the larger root under
    // the smaller and stays in the list, the others leave it.  A hook that loses
    // to a smaller one in the same pass is made again in the next, as its bond
    // is still listed.
    bool hooked = true;
    while (__syncthreads_or(hooked)) {
      hooked = false;
      bool more = true;
      while (__syncthreads_or(more)) {
        more = false;
        for (int x = threadIdx.x; x <= n; x += T) {
          const uint32_t p0 = parent[x];
          uint32_t p = p0;
          bool up = true;
#pragma unroll
          for (int h = 0; h < 4 && up; ++h) {
            const uint32_t g = parent[p];
            up = g != p;
            p = g;
          }
          if (p != p0) parent[x] = p;
          more = more || up;
        }
      }
      for (int q = threadIdx.x; q < a.nq; q += T) {
        uint32_t nib = kept[q];
        if (!nib) continue;
        const int4 b0 = __ldg(a.quad + 2 * q), b1 = __ldg(a.quad + 2 * q + 1);
        const uint32_t ends[4] = {(uint32_t)b0.x, (uint32_t)b0.z, (uint32_t)b1.x, (uint32_t)b1.z};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const uint32_t ri = parent[ends[e] & 0xFFFFu], rj = parent[ends[e] >> 16];
          if (ri == rj) nib &= ~(1u << e);
          if ((nib >> e) & 1u) atomicMin(parent + max(ri, rj), min(ri, rj));
        }
        kept[q] = (uint8_t)nib;
        hooked = hooked || nib;
      }
    }
    // 3. (the last pass hooked nothing: every link is a root)
    if (threadIdx.x == 0) dummy_root = parent[n];
    __syncthreads();
    const uint32_t rn = dummy_root;
    for (int x0 = base; x0 <= n; x0 += T) {
      const int x = x0 + lane;
      bool flip = false;
      if (x <= n) {
        const uint32_t root = parent[x];
        flip = x < n && root != rn && ((coin[root >> 5] >> (root & 31u)) & 1u);
        parent[x] = (uint32_t)x;  // for the next sweep
      }
      const uint32_t w = __ballot_sync(0xffffffffu, flip);
      if (lane == 0) sb[x0 >> 5] ^= w;
    }
    __syncthreads();
  }
  for (int x = threadIdx.x; x < n; x += T) gs[x] = ((sb[x >> 5] >> (x & 31)) & 1u) ? (int8_t)-1 : (int8_t)1;
}

// SMEM: shared memory holds parent[n + 1] (u32) | spins[n] (int8).  Otherwise
// parent is replica r's slice of gparent ([gridDim.x][n + 1]) and the spins
// are updated in place in global memory.
template <bool SMEM>
__global__ void __launch_bounds__(kSwThreads) sw_kernel(SwArgs a, uint32_t* gparent) {
  extern __shared__ __align__(16) uint32_t smem[];
  const int n = a.n;
  const int r = blockIdx.x;
  int8_t* gs = a.spins + (size_t)r * n;
  uint32_t* parent = SMEM ? smem : gparent + (size_t)r * (n + 1);
  int8_t* s = SMEM ? reinterpret_cast<int8_t*>(smem + n + 1) : gs;
  if (SMEM)
    for (int i = threadIdx.x; i < n; i += blockDim.x) s[i] = gs[i];
  const uint32_t rg = a.rep0 + (uint32_t)r;
  for (int64_t k = 0; k < a.nsweeps; ++k) {
    const float beta2 = __fmul_rn(2.0f, __ldg(a.betas + k));
    const uint32_t kk = a.sweep0 + (uint32_t)k;
    for (int i = threadIdx.x; i <= n; i += blockDim.x) parent[i] = (uint32_t)i;
    __syncthreads();
    // 1. bonds, four per thread and Philox call
    for (int e0 = 4 * threadIdx.x; e0 < a.ne; e0 += 4 * blockDim.x) {
      const ojd::u4 x = ojd::philox((uint32_t)(e0 >> 2), kk, rg, ojd::TAG_SW_BOND, a.keys);
      const uint32_t xs[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int e = e0 + q;
        if (e >= a.ne) break;
        const int i = a.ei[e], j = a.ej[e];
        const int si = s[i], sj = j < n ? s[j] : 1;
        const bool satisfied = (si * sj > 0) != (a.pos[e] != 0);  // J s_i s_j < 0
        if (satisfied && ojd::neglog(xs[q]) < __fmul_rn(beta2, a.w[e])) unite<SMEM>(parent, (uint32_t)i, (uint32_t)j);
      }
    }
    __syncthreads();
    // 2./3. roots and flips; the dummy spin's cluster stays
    const uint32_t rn = find_root<SMEM>(parent, (uint32_t)n);
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
      const uint32_t root = find_root<SMEM>(parent, (uint32_t)i);
      if (root == rn) continue;
      const ojd::u4 c = ojd::philox(root >> 2, kk, rg, ojd::TAG_SW_FLIP, a.keys);
      if (ojd::pick(c, (int)(root & 3u)) & 1u) s[i] = (int8_t)-s[i];
    }
    __syncthreads();
  }
  if (SMEM)
    for (int i = threadIdx.x; i < n; i += blockDim.x) gs[i] = s[i];
}

}  // namespace

size_t sw_smem_bytes(int n) { return (size_t)(n + 1) * 4 + (size_t)n + 16; }

namespace {

size_t sw_align(size_t b) { return (b + 255) & ~(size_t)255; }

// Shared memory of sw_hook_kernel: parent links, spin and coin bits, kept bonds.
size_t sw_hook_smem(int n, size_t nq) { return 4 * ((size_t)(n + 1) + 2 * ((size_t)(n + 32) / 32)) + (nq + 3) / 4 * 4; }

// Bytes of the separate bond arrays; the quads follow them.
size_t sw_array_bytes(size_t ne) { return 2 * sw_align(ne * 4 + 4) + sw_align(ne * 4 + 4) + sw_align(ne + 1); }

// The graph has quads: its sites are 16-bit indices and its state fits.
bool sw_has_quads(int n, size_t ne) { return n < 65535 && sw_hook_smem(n, (ne + 3) / 4) <= kSwHookSmemBytes; }

// Where the hooking kernel is the faster one (us a sweep of a 30-sweep call, energies
// included, sw_kernel / it).  A replica that has an SM to itself (1024 threads): from
// 1024 sites and 2100 bonds on (148 replicas: lattices of 32 x 32, 2048 bonds 5.8 / 6.5, and
// 33 x 33, 2178 bonds 7.8 / 7.0; 3-regular 1300 sites, 1950 bonds 6.6 / 7.2, 1400 sites
// 7.9 / 7.3).  With several replicas an SM sw_kernel's walks overlap, and they are
// short unless neighbours are near in index order, which makes long chains of sites:
// from 8192 such sites on, and with two replicas an SM from 2048 sites and 6500 bonds on
// (lattices with 256 replicas: 46 x 46 13.6 / 15.7, 56 x 56 20.2 / 20.7, 64 x 64 26.2 /
// 25.0; 1024 replicas: 64 x 64 69 / 71, 91 x 91 152 / 140); without that order only with
// two replicas an SM and four bonds a site from 2048 sites on (random, 256 replicas: 4000 sites
// of degree 8 43 / 40, 2500 of degree 20 60 / 50; but 4000 of degree 6 33.3 / 33.9), and from
// 40000 sites on (3-regular, 1024 replicas: 8200 sites 104 / 122, 20000 sites 311 / 332,
// 40000 sites 941 / 911).  Graphs that do not fit sw_kernel's shared memory: always.
bool sw_hooks(const oj_graph* g, int R, int sm_count) {
  if (!sw_has_quads(g->n, (size_t)g->sw_ne)) return false;
  if (g->n > sw_max_sites()) return true;
  if (R <= sm_count) return g->n >= 1024 && g->sw_ne >= 2100;
  if (!g->local) return g->n >= 40000 || (R <= 2 * sm_count && g->n >= 2048 && g->sw_ne >= 4 * (int64_t)g->n);
  return g->n >= 8192 || (R <= 2 * sm_count && g->n >= 2048 && g->sw_ne >= 6500);
}

}  // namespace

int sw_threads(const oj_graph* g, int R, int sm_count) {
  return sw_hooks(g, R, sm_count) && R <= sm_count ? kSwHookThreads : kSwThreads;
}

bool sw_needs_scratch(const oj_graph* g, int R, int sm_count) {
  return g->n > sw_max_sites() && !sw_hooks(g, R, sm_count);
}

// Bond list of the graph: (i, j) with i < j from the neighbour lists, then
// (i, n) for every non-zero h_i.
static cudaError_t sw_build(oj_graph* g) {
  std::vector<int32_t> ei, ej;
  std::vector<float> w;
  std::vector<uint8_t> pos;
  for (int i = 0; i < g->n; ++i)
    for (int q = g->rp[i]; q < g->rp[i + 1]; ++q) {
      const int j = g->ci[q];
      if (j <= i) continue;
      ei.push_back(i);
      ej.push_back(j);
      w.push_back((float)std::fabs(g->val64[q]));
      pos.push_back(g->val64[q] > 0 ? 1 : 0);
    }
  for (int i = 0; i < g->n; ++i)
    if (g->h64[i] != 0.0) {
      ei.push_back(i);
      ej.push_back(g->n);
      w.push_back((float)std::fabs(g->h64[i]));
      pos.push_back(g->h64[i] > 0 ? 1 : 0);
    }
  const size_t ne = ei.size();
  const size_t b_i = sw_align(ne * 4 + 4), b_w = sw_align(ne * 4 + 4), nq = (ne + 3) / 4;
  const bool quads = sw_has_quads(g->n, ne);
  cudaError_t e = g->sw_tables.ensure(sw_array_bytes(ne) + (quads ? 32 * nq : 0));
  if (e != cudaSuccess) return e;
  char* base = g->sw_tables.as<char>();
  if (quads && ne) {
    std::vector<uint32_t> quad(8 * nq, 0u);
    for (size_t b = 0; b < ne; ++b) {
      uint32_t bits;
      std::memcpy(&bits, &w[b], 4);
      quad[2 * b] = (uint32_t)ei[b] | ((uint32_t)ej[b] << 16);
      quad[2 * b + 1] = bits | (pos[b] ? 0u : 0x80000000u);
    }
    e = copy_tables(base + sw_array_bytes(ne), quad.data(), quad.size() * 4);
    if (e != cudaSuccess) return e;
  }
  if (ne) {
    if ((e = copy_tables(base, ei.data(), ne * 4)) != cudaSuccess) return e;
    if ((e = copy_tables(base + b_i, ej.data(), ne * 4)) != cudaSuccess) return e;
    if ((e = copy_tables(base + 2 * b_i, w.data(), ne * 4)) != cudaSuccess) return e;
    if ((e = copy_tables(base + 2 * b_i + b_w, pos.data(), ne)) != cudaSuccess) return e;
  }
  g->sw_ne = (int64_t)ne;
  return cudaSuccess;
}

// Builds the bond list once per graph; a host allocation that fails is
// reported as out of memory, no exception reaches the C interface.
cudaError_t sw_prepare(oj_graph* g) {
  if (g->sw_ne >= 0) return cudaSuccess;
  try {
    return sw_build(g);
  } catch (...) {
    return cudaErrorMemoryAllocation;
  }
}

cudaError_t launch_sw(const oj_graph* g, int R, int8_t* spins, const float* betas, int64_t nsweeps, RngBase rb,
                      uint32_t* scratch, int chunk, int sm_count, cudaStream_t st, int* launches) {
  const int n = g->n;
  const bool in_smem = n <= sw_max_sites();
  const size_t smem = in_smem ? sw_smem_bytes(n) : 0;
  if (g->sw_ne > (int64_t)0x7FFFFFFF || (sw_needs_scratch(g, R, sm_count) && (!scratch || chunk < 1)))
    return cudaErrorInvalidValue;
  const int64_t ne = g->sw_ne;
  const size_t b_i = sw_align((size_t)ne * 4 + 4), b_w = sw_align((size_t)ne * 4 + 4);
  const char* base = g->sw_tables.as<char>();
  SwArgs a;
  a.ei = reinterpret_cast<const int32_t*>(base);
  a.ej = reinterpret_cast<const int32_t*>(base + b_i);
  a.w = reinterpret_cast<const float*>(base + 2 * b_i);
  a.pos = reinterpret_cast<const uint8_t*>(base + 2 * b_i + b_w);
  a.quad = reinterpret_cast<const int4*>(base + sw_array_bytes((size_t)ne));
  a.nq = (int)((ne + 3) / 4);
  a.ne = (int)ne;
  a.n = n;
  a.spins = spins;
  a.betas = betas;
  a.nsweeps = nsweeps;
  a.keys = ojd::make_keys(rb.k0, rb.k1);
  a.sweep0 = rb.sweep0;
  a.rep0 = rb.rep0;
  if (sw_hooks(g, R, sm_count)) {
    const int threads = sw_threads(g, R, sm_count);
    auto kern = threads > kSwThreads ? sw_hook_kernel<kSwHookThreads, 1> : sw_hook_kernel<kSwThreads, 4>;
    const size_t hook_smem = sw_hook_smem(n, (size_t)a.nq);
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)hook_smem);
    if (e != cudaSuccess) return e;
    kern<<<R, threads, hook_smem, st>>>(a);
    if (launches) ++*launches;
    return cudaGetLastError();
  }
  if (in_smem) {
    cudaError_t e = cudaFuncSetAttribute(sw_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    sw_kernel<true><<<R, kSwThreads, smem, st>>>(a, nullptr);
    if (launches) ++*launches;
    return cudaGetLastError();
  }
  // replicas in chunks whose parent arrays fit the scratch ([chunk][n + 1])
  for (int r0 = 0; r0 < R; r0 += chunk) {
    SwArgs c = a;
    c.spins = spins + (size_t)r0 * n;
    c.rep0 = rb.rep0 + (uint32_t)r0;
    sw_kernel<false><<<std::min(chunk, R - r0), kSwThreads, 0, st>>>(c, scratch);
    if (launches) ++*launches;
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

int sw_max_sites() { return (220 * 1024 - 20) / 5; }

}  // namespace oj

// Colour-order Metropolis sweeps of small graphs whose colour classes hold
// few sites (dense QUBOs of up to a couple of hundred variables): the same
// sweeps, random numbers and FP32 operations as oj_k_colour.cu, so the same
// spins.
//
// What bounds them: the sites are a serial chain (on a complete graph every
// class is one site), and a site's field is itself a chain of n FP32 additions
// in index order, whose rounding decides the acceptance, so neither can be
// reordered.  The colour-class kernels run that chain in one thread of a CTA,
// out of global memory and with a barrier per class.  Here:
//   * the coupling matrix is dense rows in shared memory (zeros where there is
//     no coupling: adding a zero does not change a sum) and the spins are
//     +-1.0f, so a term is one FMA (v * s is exact, so it is the colour
//     kernel's addition): 4.4 cycles a term, the FMA latency;
//   * B sites are decided at once.  A group of 2^B lanes runs one chain
//     (a replica, or one Trotter slice of it); its lanes are the nodes of the
//     decision tree of the next B sites: lane 2^(d-1) + p computes the field
//     of the d-th site for the outcome p of the d - 1 sites before it (its
//     private copy of the spins holds them so), every lane tests its own
//     acceptance, and a ballot and a walk from the root give the B decisions.
//     The lanes a small call leaves idle so shorten the chain B-fold; a call
//     with many replicas takes a smaller B (seq_choose);
//   * half of the CTA's warps draw the uniforms of the next phase (Philox and
//     -ln u) into shared memory while the others sweep.
//
// Measured (one B200, one sweep, before -> now): SA on a complete graph of 64
// sites, 8 replicas 352 -> 6.0 us, 512 replicas 354 -> 6.8 us; 160 sites, 8
// replicas 2070 -> 27.5 us; SQA with 4 slices, 64 sites, 128 replicas 985 -> 11.7
// us; with 16 slices, 512 replicas 1710 -> 29.7 us.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>

#include "oj_device.cuh"
#include "oj_internal.h"

namespace oj {
namespace {

constexpr size_t kSeqSmemBytes = 220 * 1024;
constexpr int kSeqMaxSites = 256;
constexpr int kSeqMaxDepth = 5;  // largest B
constexpr int kSeqMaxWarps = 4;  // sweeping warps of a CTA (as many draw)

struct SeqArgs {
  const int32_t* rp;
  const int32_t* ci;
  const float* val;
  const float* h;
  const int32_t* order;  // sites in visiting order (by colour class)
  int n, R, T;           // T: Trotter slices (SA: 1)
  int ld;                // floats of a coupling row in shared memory
  int warps;             // sweeping warps of a CTA
  int per_cta;           // replicas of a CTA
  int8_t* spins;         // [R][T][n]
  const float* betas;    // SA: [nsweeps]
  const float2* coef;    // SQA: [nsweeps]
  int64_t nsweeps;
  ojd::Keys keys;
  uint32_t sweep0, rep0;
  unsigned long long* flips;
};

__device__ __forceinline__ float seq_terms(const float4 v, const float4 s, float f) {
  f = __fmaf_rn(v.x, s.x, f);
  f = __fmaf_rn(v.y, s.y, f);
  f = __fmaf_rn(v.z, s.z, f);
  return __fmaf_rn(v.w, s.w, f);
}

// A shared-memory load that keeps its place in the instruction stream.
__device__ __forceinline__ float4 seq_lds(uint32_t addr) {
  float4 r;
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(r.x), "=f"(r.y), "=f"(r.z), "=f"(r.w)
               : "r"(addr)
               : "memory");
  return r;
}

// Four groups of four terms: spins and couplings.
struct SeqBlock {
  float4 s[4], v[4];
};

__device__ __forceinline__ void seq_load(SeqBlock& x, uint32_t& sa, uint32_t& ra) {
#pragma unroll
  for (int g = 0; g < 4; ++g) {
    x.s[g] = seq_lds(sa + 512u * g);
    x.v[g] = seq_lds(ra + 16u * g);
  }
  sa += 2048u;
  ra += 64u;
}

// f plus the block's first `left` groups, in order; true when that was all.
__device__ __forceinline__ bool seq_step(const SeqBlock& x, int& left, float& f) {
  if (left < 4) {
    if (left > 0) f = seq_terms(x.v[0], x.s[0], f);
    if (left > 1) f = seq_terms(x.v[1], x.s[1], f);
    if (left > 2) f = seq_terms(x.v[2], x.s[2], f);
    return true;
  }
#pragma unroll
  for (int g = 0; g < 4; ++g) f = seq_terms(x.v[g], x.s[g], f);
  left -= 4;
  return left == 0;
}

// f plus ng groups of four terms, in order.  A block's loads are issued before
// the additions of the block before it (68 cycles of FMA latency, which cover
// them): 5.2 cycles a term, against 7 to 9 where the compiler places the loads
// (the ring of single groups included).  Up to seven groups past the end are
// read and not used.
__device__ __forceinline__ float seq_chain(const float* S, const float* row, int ng, float f) {
  uint32_t sa = ojd::smem_u32(S), ra = ojd::smem_u32(row);
  SeqBlock X, Y;
  seq_load(X, sa, ra);
  for (int left = ng;;) {
    seq_load(Y, sa, ra);
    if (seq_step(X, left, f)) return f;
    seq_load(X, sa, ra);
    if (seq_step(Y, left, f)) return f;
  }
}

constexpr int kSeqPad = 7 * 128;  // floats past the last spin copy that seq_chain may read

// Shared memory: table [n + B] | J [n][ld] | spins [warps][slots][ng + 1][32
// lanes][4] | L [2][n + B][chains]; ng = ceil(n / 4).  The table has, in visiting
// order, a site's place in a spin copy, its row's place in J, its field h and its
// index; it is padded with sites whose spin is in the copies' spare group and
// whose L is -infinity (never accepted), so that the last block needs no bounds.
// L holds -ln u of a phase.  Slot 0 holds the even slices (SA: the replica), slot
// 1 the odd ones; chain c of the CTA is replica c / nl, slice pair c % nl.
template <bool SQA, int B>
__global__ void __launch_bounds__(2 * kSeqMaxWarps * 32) seq_kernel(SeqArgs a) {
  extern __shared__ __align__(16) float sh[];
  constexpr int LP = B == 1 ? 1 : 1 << B;  // lanes per chain
  constexpr int CPW = 32 / LP;             // chains per warp
  const int n = a.n, ng = (n + 3) >> 2, ld = a.ld, nt = n + B;
  const int slots = SQA ? 2 : 1, sstride = (ng + 1) * 128, W = a.warps;
  const int T = a.T;
  const int nl = SQA ? (T + 1) >> 1 : 1;  // chains per replica
  const int r0 = blockIdx.x * a.per_cta;
  const int nrep = min(a.per_cta, a.R - r0);
  const int nchain = a.per_cta * nl;
  int4* tab = reinterpret_cast<int4*>(sh);
  float* J = sh + 4 * nt;
  float* Sp = J + (size_t)n * ld;
  float* Lb = Sp + (size_t)W * slots * sstride + kSeqPad;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int e = threadIdx.x; e < n * ld; e += blockDim.x) J[e] = 0.0f;
  for (int e = threadIdx.x; e < nt; e += blockDim.x) {
    const int i = e < n ? a.order[e] : 4 * ng;
    tab[e] = make_int4((i >> 2) * 128 + (i & 3), e < n ? i * ld : 0, e < n ? __float_as_int(a.h[i]) : 0, i);
  }
  for (int e = threadIdx.x; e < 2 * nt * nchain; e += blockDim.x) Lb[e] = -INFINITY;
  __syncthreads();
  for (int i = warp; i < n; i += 2 * W)
    for (int p = a.rp[i] + lane; p < a.rp[i + 1]; p += 32) J[i * ld + a.ci[p]] = a.val[p];
  // this lane's chain (sweeping warps): replica rl, slices 2m and 2m + 1
  const int chain = (warp < W ? warp : 0) * CPW + lane / LP;
  const int rl = chain / nl, m = chain - rl * nl;
  const bool live = warp < W && rl < nrep;
  float* Sw = Sp + (size_t)(warp < W ? warp : 0) * slots * sstride + 4 * lane;
  if (warp < W)
    for (int sl = 0; sl < slots; ++sl) {
      const int t = 2 * m + sl;
      const bool on = live && t < T;
      const int8_t* gs = a.spins + ((size_t)(r0 + (on ? rl : 0)) * T + (on ? t : 0)) * n;
#pragma unroll 8
      for (int i = 0; i < 4 * ng + 4; ++i)
        Sw[sl * sstride + (i >> 2) * 128 + (i & 3)] = on && i < n && gs[i] < 0 ? -1.0f : 1.0f;
    }
  const int nph = SQA ? ((T & 1) ? 3 : 2) : 1;  // phases of a sweep: slice groups
  const int64_t total = a.nsweeps * nph;
  // -ln u of one phase: every site and chain
  auto draw = [&](int64_t k, int grp, float* L, int tid, int nthr) {
    const uint32_t kk = a.sweep0 + (uint32_t)k;
    if constexpr (!SQA) {
      const int qlo = r0 >> 2, nq = ((r0 + nrep + 3) >> 2) - qlo;
      for (int it = tid; it < n * nq; it += nthr) {
        const int idx = it / nq, q = qlo + it - idx * nq;
        const ojd::u4 x = ojd::philox((uint32_t)tab[idx].w, kk, (a.rep0 >> 2) + (uint32_t)q, ojd::TAG_SA, a.keys);
        float* o = L + idx * nchain - r0;
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (4 * q + j >= r0 && 4 * q + j < r0 + nrep) o[4 * q + j] = ojd::neglog(ojd::pick(x, j));
      }
    } else {
      const int nq = (nl + 3) >> 2, per = nrep * nq;
      const uint32_t par = grp == 1 ? 1u : 0u;
      for (int it = tid; it < n * per; it += nthr) {
        const int idx = it / per, rq = it - idx * per, r = rq / nq, q = rq - r * nq;
        const ojd::u4 x = ojd::philox((uint32_t)tab[idx].w, kk, a.rep0 + (uint32_t)(r0 + r),
                                      ((uint32_t)q << 9) | (par << 8) | ojd::TAG_SQA, a.keys);
        float* o = L + idx * nchain + r * nl + 4 * q;
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (4 * q + j < nl) o[j] = ojd::neglog(ojd::pick(x, j));
      }
    }
  };
  if (total > 0) draw(0, 0, Lb, threadIdx.x, blockDim.x);
  __syncthreads();
  // this lane's node of the decision tree: depth d, and whether the sites
  // before it (first site: highest bit) are flipped on its path
  const int node = B == 1 ? 1 : max(lane & (LP - 1), 1);
  const int depth = 32 - __clz(node);
  const bool root = B == 1 || (lane & (LP - 1)) == 1;  // the lane that counts the chain's flips
  uint32_t path[B];  // sign bits of the flips on the path
#pragma unroll
  for (int d = 0; d < B; ++d) path[d] = d + 1 < depth && ((node >> (depth - 2 - d)) & 1) ? 0x80000000u : 0u;
  unsigned long long nflip = 0;
  int64_t k = 0, kn = 0;  // this phase's sweep and slice group, the next phase's
  int grp = 0, gn = 0;
  float2 par = make_float2(0.0f, 0.0f);
  if (total > 0) par = SQA ? a.coef[0] : make_float2(2.0f * a.betas[0], 0.0f);
  for (int64_t ph = 0; ph < total; ++ph) {
    if (++gn == nph) {
      gn = 0;
      ++kn;
    }
    if (warp >= W) {
      if (ph + 1 < total)
        draw(kn, gn, Lb + (size_t)((ph + 1) & 1) * nt * nchain, threadIdx.x - 32 * W, blockDim.x - 32 * W);
    } else {
      float2 pnext = par;  // the next phase's coefficients are in flight during this one
      if (kn != k && kn < a.nsweeps) pnext = SQA ? __ldg(a.coef + kn) : make_float2(2.0f * __ldg(a.betas + kn), 0.0f);
      const float* L = Lb + (size_t)(ph & 1) * nt * nchain + min(chain, nchain - 1);
      const int sl = SQA && grp == 1 ? 1 : 0;
      float* S = Sw + sl * sstride;
      bool on = live;
      // the slice's Trotter neighbours t + 1 and t - 1 (periodic in T), in
      // their own chains' copies; they do not change during this phase
      const float *Su = S, *Sd = S;
      if constexpr (SQA) {
        const int t = 2 * m + sl;
        on = live && t < T && ((T & 1) ? (grp == 2 ? t == T - 1 : t < T - 1) : true);
        const int tu = t + 1 >= T ? 0 : t + 1, td = t == 0 ? T - 1 : t - 1;
        const int cu = on ? rl * nl + (tu >> 1) : chain, cd = on ? rl * nl + (td >> 1) : chain;
        Su = Sp + ((size_t)(cu / CPW) * slots + (tu & 1)) * sstride + 4 * (cu % CPW) * LP;
        Sd = Sp + ((size_t)(cd / CPW) * slots + (td & 1)) * sstride + 4 * (cd % CPW) * LP;
      }
      // the next B sites' places in the copy and spins, and this lane's own
      // site; fetched after the block before is decided and stored, so that this
      // latency is part of every block's chain
      uint32_t* Sb = reinterpret_cast<uint32_t*>(S);
      int o[B];
      uint32_t v[B];
      float hi, Li, su = 0.0f, sd = 0.0f;
      uint32_t si;
      const float* row;
      auto fetch = [&](int idx) {
#pragma unroll
        for (int d = 0; d < B; ++d) o[d] = tab[idx + d].x;
        const int4 e = tab[idx + depth - 1];
        Li = L[(idx + depth - 1) * nchain];
        row = J + e.y;
        hi = __int_as_float(e.z);
#pragma unroll
        for (int d = 0; d < B; ++d) v[d] = Sb[o[d]];
        si = Sb[e.x];
        if constexpr (SQA) {
          su = Su[e.x];
          sd = Sd[e.x];
        }
      };
      fetch(0);
      for (int idx = 0; idx < n; idx += B) {
        // the path's flips in this lane's copy
#pragma unroll
        for (int d = 0; d + 1 < B; ++d) Sb[o[d]] = v[d] ^ path[d];
        const float f = seq_chain(S, row, ng, hi);
        bool acc;
        if constexpr (SQA) {
          // -2 s f and -2 s (s' + s''), s the sign of the spin
          const float dEsp = __uint_as_float(__float_as_uint(-2.0f * f) ^ (si & 0x80000000u));
          const float dEtrot = __uint_as_float(__float_as_uint(-2.0f * (su + sd)) ^ (si & 0x80000000u));
          acc = __fadd_rn(__fmul_rn(par.x, dEsp), __fmul_rn(par.y, dEtrot)) < Li;
        } else {
          const float bf = __fmul_rn(par.x, f);
          acc = __uint_as_float(__float_as_uint(-bf) ^ (si & 0x80000000u)) < Li;
        }
        acc = acc && on;
        uint32_t w = 1u;  // the walk from the root: bit B - 1 - d is the decision of site d
        if constexpr (B == 1) {
          w = acc ? 3u : 2u;
        } else {
          const uint32_t bits = __ballot_sync(0xffffffffu, acc) >> (lane & ~(LP - 1));
#pragma unroll
          for (int d = 0; d < B; ++d) w = 2u * w + ((bits >> w) & 1u);
        }
#pragma unroll
        for (int d = 0; d < B; ++d) Sb[o[d]] = v[d] ^ ((w << (32 - B + d)) & 0x80000000u);
        if (root) nflip += __popc(w) - 1;
        fetch(min(idx + B, n));
      }
      par = pnext;
    }
    k = kn;
    grp = gn;
    __syncthreads();
  }
  if (warp < W && live && (lane & (LP - 1)) == 0)
    for (int sl = 0; sl < slots; ++sl) {
      const int t = 2 * m + sl;
      if (t >= T) break;
      int8_t* gs = a.spins + ((size_t)(r0 + rl) * T + t) * n;
#pragma unroll 8
      for (int i = 0; i < n; ++i) gs[i] = Sw[sl * sstride + (i >> 2) * 128 + (i & 3)] < 0.0f ? (int8_t)-1 : (int8_t)1;
    }
  if (warp < W) ojd::add_flips(a.flips, nflip);
}

// Floats of a row: a multiple of four, an odd number of 16-byte units, so that
// the rows of consecutive sites lie in different banks.
int seq_ld(int n) {
  const int ng = (n + 3) / 4;
  return 4 * (ng | 1);
}

struct SeqShape {
  int B = 0, warps = 0, per_cta = 0;
  size_t smem = 0;
};

size_t seq_smem_bytes(int n, int T, int warps, int chains) {
  const size_t ng = (size_t)(n + 3) / 4, slots = T > 1 ? 2 : 1, nt = (size_t)n + kSeqMaxDepth;
  return 4 * (4 * nt + (size_t)n * seq_ld(n) + (size_t)warps * slots * (ng + 1) * 128 + kSeqPad +
              2 * nt * chains);
}

// The shape with B lanes' depth for T slices: whole replicas per CTA.
SeqShape seq_shape(int n, int T, int B, int warps) {
  SeqShape s;
  const int cpw = B == 1 ? 32 : 32 >> B, nl = T > 1 ? (T + 1) / 2 : 1;
  s.B = B;
  s.warps = std::max(warps, (nl + cpw - 1) / cpw);
  s.per_cta = s.warps * cpw / nl;
  s.smem = seq_smem_bytes(n, T, s.warps, s.per_cta * nl);
  if (s.warps > kSeqMaxWarps || s.smem > kSeqSmemBytes) s.B = 0;
  return s;
}

// The deepest tree whose sweeping warps still get a scheduler each (four per
// SM) and whose CTAs are all resident; a call with more replicas than that is
// bound by issue slots, where one lane per chain does the least work.
SeqShape seq_choose(int n, int T, int R, int sm_count) {
  for (int B = kSeqMaxDepth; B >= 2; --B) {
    const SeqShape s = seq_shape(n, T, B, 1);
    if (!s.B) continue;
    const int64_t ctas = (R + s.per_cta - 1) / s.per_cta;
    const int64_t resident = (int64_t)sm_count * std::min<int64_t>(4, (int64_t)(224 * 1024) / (int64_t)(s.smem + 1024));
    if (ctas <= resident && ctas * s.warps <= 4LL * sm_count) return s;
  }
  for (int w = 4; w >= 1; w /= 2) {
    const SeqShape s = seq_shape(n, T, 1, w);
    if (s.B && (w == 1 || (R + s.per_cta - 1) / s.per_cta >= sm_count)) return s;
  }
  return SeqShape{};
}

template <bool SQA>
cudaError_t launch_seq(const oj_graph* g, int R, int T, int8_t* spins, const float* betas, const float2* coef,
                       int64_t nsweeps, RngBase rb, cudaStream_t st, int* launches) {
  int sms = 0;
  cudaError_t e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, g->device);
  if (e != cudaSuccess) return e;
  const SeqShape sp = seq_choose(g->n, T, R, sms);
  SeqArgs a;
  a.rp = g->d_rp.as<int32_t>();
  a.ci = g->d_ci.as<int32_t>();
  a.val = g->d_val.as<float>();
  a.h = g->d_h.as<float>();
  a.order = g->d_order.as<int32_t>();
  a.n = g->n;
  a.R = R;
  a.T = T;
  a.ld = seq_ld(g->n);
  a.warps = sp.warps;
  a.per_cta = sp.per_cta;
  a.spins = spins;
  a.betas = betas;
  a.coef = coef;
  a.nsweeps = nsweeps;
  a.keys = ojd::make_keys(rb.k0, rb.k1);
  a.sweep0 = rb.sweep0;
  a.rep0 = rb.rep0;
  a.flips = rb.flips;
  auto go = [&](auto kern) {
    e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sp.smem);
    if (e != cudaSuccess) return e;
    kern<<<(R + sp.per_cta - 1) / sp.per_cta, 64 * sp.warps, sp.smem, st>>>(a);
    if (launches) ++*launches;
    return cudaGetLastError();
  };
  switch (sp.B) {
    case 1: return go(seq_kernel<SQA, 1>);
    case 2: return go(seq_kernel<SQA, 2>);
    case 3: return go(seq_kernel<SQA, 3>);
    case 4: return go(seq_kernel<SQA, 4>);
    case 5: return go(seq_kernel<SQA, 5>);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace

// A graph goes through the serial kernel when its matrix, spins and uniforms
// fit shared memory and a sweep is shorter there.  Cycles of a sweep: about
// n (85 + 1.6 n) here (five sites at once), 850 + 55 deg per class in the
// colour-class kernels.  Measured near the line (SA with 8 replicas, us a sweep
// there / here): 48 sites, 6 classes of mean degree 10: 4.5 / 3.8; 64 sites, 15
// classes of degree 32: 17.9 / 6.1; 64 sites, 8 classes of degree 13: 6.2 / 6.1, but
// with 512 replicas 6.3 / 7.0 (stays there); 100 sites, 11 classes of degree 20:
// 10.9 / 12.7 (stays there).
bool seq_applies(const oj_graph* g, int T) {
  const double n = g->n;
  if (g->n < 1 || g->n > kSeqMaxSites || !seq_shape(g->n, T, 1, 1).B) return false;
  return n * (85.0 + 1.6 * n) < 0.95 * g->info.num_colours * (850.0 + 55.0 * (double)g->info.nnz / n);
}

cudaError_t launch_sa_seq(const oj_graph* g, int R, int8_t* spins, const float* betas, int64_t nsweeps, RngBase rb,
                          cudaStream_t st, int* launches) {
  return launch_seq<false>(g, R, 1, spins, betas, nullptr, nsweeps, rb, st, launches);
}

cudaError_t launch_sqa_seq(const oj_graph* g, int R, int T, int8_t* spins, const float2* coef, int64_t nsweeps,
                           RngBase rb, cudaStream_t st, int* launches) {
  return launch_seq<true>(g, R, T, spins, nullptr, coef, nsweeps, rb, st, launches);
}

}  // namespace oj

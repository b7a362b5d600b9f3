// Colour-class Metropolis kernels for arbitrary coupling graphs (FP32 fields
// gathered from the neighbour list), the FP64 energy kernel and the
// int8 <-> bit-packed conversion kernels.
//
// SA (reference: include/openjij/updater/single_spin_flip.hpp:66-95).  The
// reference visits sites 0..n-1 in order.  Here the sites are split into the
// classes of a greedy colouring of the coupling graph; sites of one class have
// no coupling between them, so a whole class is updated at once and classes
// are visited in order.  On a 2-colourable lattice this is the checkerboard
// sweep; on a complete graph every class is a single site and the order is the
// reference's.  Acceptance: dE <= 0, or beta*dE < -ln(u) (equivalent to
// exp(-beta*dE) > u, single_spin_flip.hpp:80-82).
//
// SQA (single_spin_flip.hpp:127-258): slice groups {even t < T - T%2}, {odd t},
// {T-1 if T odd} in that order as the reference's OpenMP loops, and inside a
// group the colour classes of the spatial graph.  dE = a*dE_sp + B*dE_trot with
// a = s*beta/T and B = 0.5*log(tanh(beta*Gamma*(1-s)/T)) precomputed per sweep;
// accept when dE < -ln(u) (single_spin_flip.hpp:240: dE < 0 || exp(-dE) > u).
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cstring>
#include <memory>
#include <vector>

#include "oj_device.cuh"
#include "oj_internal.h"

namespace oj {
namespace {

// Most threads of a CTA with the spins in shared memory.  An SM has 1024 at work
// (colour_threads), so the kernels ask for one CTA an SM of this size, 64 registers a
// thread; with the bound of threads alone the compiler took 32, which put the loads
// of a neighbour list one after another (300 sites of mean degree 90, 31 classes, us a
// sweep: SA with 8 replicas 577, now 114; SQA with 2 slices 692, now 195; 300 sites of
// degree 4, SA with 8 replicas 9.5, now 6.5).
constexpr int kColourThreads = 1024;
constexpr int kColourGlobalThreads = 256;  // SA with the spins in global memory
constexpr int kSqaGlobalThreads = 512;     // SQA with the spins in global memory
constexpr int kSmemBudget = 200 * 1024;

// Arguments of the kernels with the spins in shared memory (ColourPlan tables).
struct ColourArgs {
  const int2* site;
  const int4* cls;
  const int2* slice;
  const int2* ent;
  int ncol, n, R, T;
  int8_t* spins;        // [R][T][n]
  const float* betas;   // SA: [nsweeps]
  const float2* coef;   // SQA: [nsweeps]
  int64_t nsweeps;
  ojd::Keys keys;
  uint32_t sweep0, rep0;
  unsigned long long* flips;
};

// Adds the neighbours' couplings of this lane's slot to NF fields, in neighbour
// order.  S: one byte per slot; field q takes the sign of its spin from bit
// b0 + q STEP of the neighbour's byte (set: -1).  The terms of a slice are the
// same for the whole warp; width: the slice's slots.  LONG: 16 entries in flight
// (they come from L2 on graphs with long lists).
template <int NF, int STEP, bool LONG>
__device__ __forceinline__ void colour_fields(const int2* __restrict__ ent, int terms, int width,
                                              const uint8_t* __restrict__ S, int b0, float (&f)[NF]) {
  const int sh = 31 - (NF - 1) * STEP - b0;
  auto add = [&](const int2 e) {
    const uint32_t w = (uint32_t)S[e.x] << sh;
#pragma unroll
    for (int q = 0; q < NF; ++q)
      f[q] = __fadd_rn(f[q], __uint_as_float((uint32_t)e.y ^ ((w << ((NF - 1 - q) * STEP)) & 0x80000000u)));
  };
  int p = 0;
  if constexpr (LONG) {
    for (; p + 16 <= terms; p += 16) {
      int2 e[16];
#pragma unroll
      for (int q = 0; q < 16; ++q) e[q] = __ldg(ent + width * (p + q));
#pragma unroll
      for (int q = 0; q < 16; ++q) add(e[q]);
    }
  }
  if (!LONG && width == 32) {  // a full slice: constant offsets
#pragma unroll 4
    for (; p < terms; ++p) add(__ldg(ent + 32 * p));
  } else {
#pragma unroll 4
    for (; p < terms; ++p) add(__ldg(ent + width * p));
  }
}

// SA, the spins in shared memory.  What bounds the sweep is the issue rate:
// per attempt the kernel had about 112 instructions (four byte loads, compares
// and selects per neighbour and replica quad, 17 for -ln u), half the slots
// busy, the rest waiting on dependent loads (order, row pointers, columns).
// Here a CTA runs 4 NQ replicas, their spins at a site in the bits of one byte:
// a neighbour is one coalesced 8-byte entry and one byte load for all of them,
// and a shift, a logic operation and an addition per replica; the acceptance
// takes the hardware logarithm and calls neglog only when that is too close
// to tell (neglog_gap).  Chimera lattice of 2048
// sites with fields, 1024 replicas, 1000 sweeps: 11.97 -> 5.02 ms (56 instructions an attempt, ALU pipe 63 %).
template <int NQ, bool LONG>
__global__ void __launch_bounds__(kColourThreads, 1) sa_colour_kernel(ColourArgs a) {
  extern __shared__ uint8_t S[];  // [n] by slot
  constexpr int NF = 4 * NQ;
  const int r0 = NF * blockIdx.x, nr = min(NF, a.R - r0);
  const int n = a.n;
  const uint32_t valid = (1u << nr) - 1u;
  int8_t* gs = a.spins + (size_t)r0 * n;
  for (int idx = threadIdx.x; idx < n; idx += blockDim.x) {
    const int i = a.site[idx].x;
    uint32_t w = 0u;
    for (int r = 0; r < nr; ++r)
      if (gs[(size_t)r * n + i] < 0) w |= 1u << r;
    S[idx] = (uint8_t)w;
  }
  __syncthreads();
  const uint32_t quad0 = (a.rep0 >> 2) + (uint32_t)(NQ * blockIdx.x);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = blockDim.x >> 5;
  unsigned long long nflip = 0;
  float beta2 = a.nsweeps > 0 ? 2.0f * __ldg(a.betas) : 0.0f;
  for (int64_t k = 0; k < a.nsweeps; ++k) {
    const float bnext = k + 1 < a.nsweeps ? 2.0f * __ldg(a.betas + k + 1) : 0.0f;
    const uint32_t kk = a.sweep0 + (uint32_t)k;
    for (int c = 0; c < a.ncol; ++c) {
      const int4 cl = __ldg(a.cls + c);
      for (int sl = warp; 32 * sl < cl.y; sl += nwarps) {
        const int2 sd = __ldg(a.slice + cl.z + sl);
        const int idx = cl.x + 32 * sl + lane;
        const int width = min(32, cl.y - 32 * sl);
        if (lane >= width) continue;
        const int2 site = __ldg(a.site + idx);
        uint32_t x[NF];
#pragma unroll
        for (int q = 0; q < NQ; ++q) {
          const ojd::u4 u = ojd::philox((uint32_t)site.x, kk, quad0 + (uint32_t)q, ojd::TAG_SA, a.keys);
          x[4 * q] = u.x;
          x[4 * q + 1] = u.y;
          x[4 * q + 2] = u.z;
          x[4 * q + 3] = u.w;
        }
        float f[NF];
#pragma unroll
        for (int q = 0; q < NF; ++q) f[q] = __int_as_float(site.y);
        const uint32_t w = S[idx];
        colour_fields<NF, 1, LONG>(a.ent + sd.x + lane, sd.y, width, S, 0, f);
        // beta*dE, dE = -+2 f, is (2 beta) f with the sign of -s_i (scaling by
        // 2 is exact); dE <= 0 accepts without a draw, and so does the
        // comparison, since -ln u > 0 and beta is finite and >= 0
        uint32_t flip = 0u;
        bool near = false;
#pragma unroll
        for (int q = 0; q < NF; ++q) {
          f[q] = __uint_as_float(__float_as_uint(__fmul_rn(beta2, f[q])) ^ ((~w << (31 - q)) & 0x80000000u));
          const float t = ojd::neglog_gap(f[q], x[q]);
          if (t < 0.0f) flip |= 1u << q;
          near = near || fabsf(t) <= ojd::kNegLogTol;
        }
        if (near) {
          flip = 0u;
#pragma unroll
          for (int q = 0; q < NF; ++q)
            if (f[q] < ojd::neglog(x[q])) flip |= 1u << q;
        }
        S[idx] = (uint8_t)(w ^ flip);
        nflip += __popc(flip & valid);
      }
      __syncthreads();
    }
    beta2 = bnext;
  }
  for (int idx = threadIdx.x; idx < n; idx += blockDim.x) {
    const int i = a.site[idx].x;
    const uint32_t w = S[idx];
    for (int r = 0; r < nr; ++r) gs[(size_t)r * n + i] = ((w >> r) & 1u) ? (int8_t)-1 : (int8_t)1;
  }
  ojd::add_flips(a.flips, nflip);
}

// SQA, the spins in shared memory: one CTA per replica, one thread per (slot,
// octet of slices), which updates the octet's up to NJ slices of the active
// parity.  The octet's spins are the bits of one byte, read and written whole
// by its own thread; its other parity and the neighbouring octets' edge bits
// do not change during the phase.  The same field, random number and acceptance
// steps as the SA kernel above.  Chimera lattice of 512 sites,
// 8 slices, 128 replicas, 500 sweeps: 5.11 -> 1.94 ms.
template <int NJ, bool LONG>
__global__ void __launch_bounds__(kColourThreads, 1) sqa_colour_kernel(ColourArgs a) {
  extern __shared__ uint8_t S[];  // [octets][n] by slot
  const int r = blockIdx.x;
  const int n = a.n, T = a.T, no = (T + 7) >> 3;
  int8_t* gs = a.spins + (size_t)r * T * n;
  for (int it = threadIdx.x; it < n * no; it += blockDim.x) {
    const int o = it / n, idx = it - o * n;
    const int i = a.site[idx].x;
    uint32_t w = 0u;
    for (int q = 0; q < 8 && 8 * o + q < T; ++q)
      if (gs[(size_t)(8 * o + q) * n + i] < 0) w |= 1u << q;
    S[it] = (uint8_t)w;
  }
  __syncthreads();
  const uint32_t rg = a.rep0 + (uint32_t)r;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = blockDim.x >> 5;
  const int upper = T & ~1, last = 8 * (no - 1);
  unsigned long long nflip = 0;
  float2 ab = a.nsweeps > 0 ? __ldg(a.coef) : make_float2(0.0f, 0.0f);
  for (int64_t k = 0; k < a.nsweeps; ++k) {
    const float2 abnext = k + 1 < a.nsweeps ? __ldg(a.coef + k + 1) : ab;
    const uint32_t kk = a.sweep0 + (uint32_t)k;
    // slice groups: the even slices below upper, the odd ones, slice T - 1 when
    // T is odd
    for (int grp = 0; grp < ((T & 1) ? 3 : 2); ++grp) {
      const int par = grp == 1 ? 1 : 0;
      const int o0 = grp == 2 ? no - 1 : 0;
      const int on = grp == 2 ? 1 : (upper - par + 7) >> 3;  // octets with a slice of the group
      for (int c = 0; c < a.ncol; ++c) {
        const int4 cl = __ldg(a.cls + c);
        const int ns = (cl.y + 31) >> 5;
        for (int ws = warp; ws < ns * on; ws += nwarps) {
          const int oo = on == 1 ? 0 : ws / ns, sl = ws - oo * ns;
          const int o = o0 + oo;
          const int2 sd = __ldg(a.slice + cl.z + sl);
          const int idx = cl.x + 32 * sl + lane;
          const int width = min(32, cl.y - 32 * sl);
          if (lane >= width) continue;
          const int2 site = __ldg(a.site + idx);
          const ojd::u4 u = ojd::philox((uint32_t)site.x, kk, rg,
                                        ((uint32_t)o << 9) | ((uint32_t)par << 8) | ojd::TAG_SQA, a.keys);
          float f[NJ];
#pragma unroll
          for (int j = 0; j < NJ; ++j) f[j] = __int_as_float(site.y);
          uint8_t* So = S + (size_t)o * n;
          const uint32_t w = So[idx];
          colour_fields<NJ, 2, LONG>(a.ent + sd.x + lane, sd.y, width, So, par, f);
          // bit q + 1 of the window is slice 8 o + q; below and above it the
          // slices before and after, periodic in T
          const uint32_t before = o ? (uint32_t)So[idx - n] >> 7
                                    : (uint32_t)S[(size_t)(no - 1) * n + idx] >> (T - 1 - last);
          uint32_t win = (w << 1) | (before & 1u);
          if (o == no - 1)
            win |= ((uint32_t)S[idx] & 1u) << (T - last + 1);
          else
            win |= ((uint32_t)So[idx + n] & 1u) << 9;
          uint32_t flip = 0u;
          bool near = false;
#pragma unroll
          for (int j = 0; j < NJ; ++j) {
            const uint32_t v = win >> (2 * j + par);  // bits 0, 1, 2: slices t - 1, t, t + 1
            // -2 s_t f and -2 s_t (s_{t+1} + s_{t-1}): 2 where a neighbour differs, -2 where it is the same
            const float dEsp = __uint_as_float(__float_as_uint(2.0f * f[j]) ^ ((~v << 30) & 0x80000000u));
            const float dn = __uint_as_float(0xC0000000u ^ (((v ^ (v >> 1)) << 31) & 0x80000000u));
            const float up = __uint_as_float(0xC0000000u ^ (((v ^ (v >> 1)) << 30) & 0x80000000u));
            f[j] = __fadd_rn(__fmul_rn(ab.x, dEsp), __fmul_rn(ab.y, dn + up));
            const float t = ojd::neglog_gap(f[j], ojd::pick(u, j));
            if (t < 0.0f) flip |= 1u << (2 * j);
            near = near || fabsf(t) <= ojd::kNegLogTol;
          }
          if (near) {
            flip = 0u;
#pragma unroll
            for (int j = 0; j < NJ; ++j)
              if (f[j] < ojd::neglog(ojd::pick(u, j))) flip |= 1u << (2 * j);
          }
          // the slices of the group in this octet
          uint32_t act = 0x55u << par;
          if (grp == 2)
            act = 1u << (T - 1 - last);
          else if (8 * o + 8 > upper)
            act &= (1u << (upper - 8 * o)) - 1u;
          flip = (flip << par) & act;
          So[idx] = (uint8_t)(w ^ flip);
          nflip += __popc(flip);
        }
        __syncthreads();
      }
    }
    ab = abnext;
  }
  for (int it = threadIdx.x; it < n * no; it += blockDim.x) {
    const int o = it / n, idx = it - o * n;
    const int i = a.site[idx].x;
    const uint32_t w = S[it];
    for (int q = 0; q < 8 && 8 * o + q < T; ++q)
      gs[(size_t)(8 * o + q) * n + i] = ((w >> q) & 1u) ? (int8_t)-1 : (int8_t)1;
  }
  ojd::add_flips(a.flips, nflip);
}

// SA on graphs whose spins do not fit shared memory, or whose tables
// (ColourPlan) there is no room for; the spins are updated in place in global
// memory.  One CTA per replica quad q (replicas 4q..4q+3); one thread per
// (site, quad): the four replicas share the neighbour loads and one Philox call.
__global__ void __launch_bounds__(kColourGlobalThreads)
    sa_colour_global_kernel(const int32_t* __restrict__ rp, const int32_t* __restrict__ ci,
                     const float* __restrict__ val, const float* __restrict__ h,
                     const int32_t* __restrict__ order, const int32_t* __restrict__ coff, int ncol,
                     int n, int R, int8_t* __restrict__ spins, const float* __restrict__ betas,
                     int64_t nsweeps, RngBase rb) {
  const int q = blockIdx.x;
  const int r0 = 4 * q;
  const int nr = min(4, R - r0);
  int8_t* S = spins + (size_t)r0 * n;
  unsigned long long nflip = 0;
  for (int64_t k = 0; k < nsweeps; ++k) {
    const float beta2 = 2.0f * betas[k];
    for (int c = 0; c < ncol; ++c) {
      const int lo = coff[c], hi = coff[c + 1];
      for (int idx = lo + threadIdx.x; idx < hi; idx += blockDim.x) {
        const int i = order[idx];
        const float hi_f = h[i];
        float f0 = hi_f, f1 = hi_f, f2 = hi_f, f3 = hi_f;
        const int p1 = rp[i + 1];
        for (int p = rp[i]; p < p1; ++p) {
          const int j = ci[p];
          const float v = val[p];
          f0 = __fadd_rn(f0, S[j] > 0 ? v : -v);
          if (nr > 1) f1 = __fadd_rn(f1, S[n + j] > 0 ? v : -v);
          if (nr > 2) f2 = __fadd_rn(f2, S[2 * n + j] > 0 ? v : -v);
          if (nr > 3) f3 = __fadd_rn(f3, S[3 * n + j] > 0 ? v : -v);
        }
        const ojd::u4 rnd = ojd::philox((uint32_t)i, rb.sweep0 + (uint32_t)k, (rb.rep0 >> 2) + (uint32_t)q,
                                        ojd::TAG_SA, rb.k0, rb.k1);
        const float fs[4] = {f0, f1, f2, f3};
#pragma unroll
        for (int rl = 0; rl < 4; ++rl) {
          if (rl < nr) {
            const int8_t si = S[rl * n + i];
            // beta*dE, dE = -+2 f, is (2 beta) f with the sign of -s_i (scaling
            // by 2 is exact); dE <= 0 accepts without a draw, and so does the
            // comparison, since -ln u > 0 and beta is finite and >= 0
            const float bf = __fmul_rn(beta2, fs[rl]);
            if ((si > 0 ? -bf : bf) < ojd::neglog(ojd::pick(rnd, rl))) {
              S[rl * n + i] = (int8_t)(-si);
              ++nflip;
            }
          }
        }
      }
      __syncthreads();
    }
  }
  ojd::add_flips(rb.flips, nflip);
}

// SQA likewise: one CTA per replica; one thread per (site, slice quad) of the
// active group.
__global__ void __launch_bounds__(kSqaGlobalThreads)
    sqa_colour_global_kernel(const int32_t* __restrict__ rp, const int32_t* __restrict__ ci,
                      const float* __restrict__ val, const float* __restrict__ h,
                      const int32_t* __restrict__ order, const int32_t* __restrict__ coff, int ncol,
                      int n, int T, int8_t* __restrict__ spins, const float2* __restrict__ coef,
                      int64_t nsweeps, RngBase rb) {
  const int r = blockIdx.x;
  const size_t tn = (size_t)T * n;
  int8_t* S = spins + (size_t)r * tn;
  unsigned long long nflip = 0;
  const int upper = (T & 1) ? T - 1 : T;
  const int nquad = (T + 7) >> 3;
  for (int64_t k = 0; k < nsweeps; ++k) {
    const float2 ab = coef[k];
    for (int grp = 0; grp < 3; ++grp) {
      if (grp == 2 && !(T & 1)) break;
      const int par = grp == 1 ? 1 : 0;
      const int tmin = grp == 2 ? T - 1 : 0;
      const int tmax = grp == 0 ? upper : T;  // exclusive
      for (int c = 0; c < ncol; ++c) {
        const int lo = coff[c], cnt = coff[c + 1] - lo;
        const int items = cnt * nquad;
        for (int it = threadIdx.x; it < items; it += blockDim.x) {
          const int a = it / cnt;
          const int i = order[lo + (it - a * cnt)];
          const int tq = 8 * a + par;
          if (tq + 6 < tmin || tq >= tmax) continue;
          const ojd::u4 rnd = ojd::philox((uint32_t)i, rb.sweep0 + (uint32_t)k, rb.rep0 + (uint32_t)r,
                                          ((uint32_t)a << 9) | ((uint32_t)par << 8) | ojd::TAG_SQA,
                                          rb.k0, rb.k1);
          const float hi_f = h[i];
          const int p0 = rp[i], p1 = rp[i + 1];
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const int t = tq + 2 * j;
            if (t < tmin || t >= tmax) continue;
            int8_t* St = S + (size_t)t * n;
            float f = hi_f;
            for (int p = p0; p < p1; ++p) {
              const float v = val[p];
              f = __fadd_rn(f, St[ci[p]] > 0 ? v : -v);
            }
            const int8_t si = St[i];
            const float dEsp = si > 0 ? -2.0f * f : 2.0f * f;
            const int tp = t + 1 == T ? 0 : t + 1;
            const int tm = t == 0 ? T - 1 : t - 1;
            const int ssum = (int)S[(size_t)tp * n + i] + (int)S[(size_t)tm * n + i];
            const float dEtrot = (float)(-2 * (int)si * ssum);
            const float dE = __fadd_rn(__fmul_rn(ab.x, dEsp), __fmul_rn(ab.y, dEtrot));
            const float L = ojd::neglog(ojd::pick(rnd, j));
            if (dE < L) {
              St[i] = (int8_t)(-si);
              ++nflip;
            }
          }
        }
        __syncthreads();
      }
    }
  }
  ojd::add_flips(rb.flips, nflip);
}

// FP64 energies of 32 spin vectors per CTA:
// E = sum_{i<j} J_ij s_i s_j + sum_i h_i s_i  (= dense.hpp:176-192).
// The 32 vectors' spins at a site are packed into one word (bit r set iff
// s = -1), so every coupling is read once for 32 vectors and s_i s_j is the
// xor of two words.  Partial sums are combined in a fixed order, so the result
// does not depend on timing.
constexpr int kEnergyThreads = 256;
__global__ void __launch_bounds__(kEnergyThreads)
    energy_kernel(const int32_t* __restrict__ rp, const int32_t* __restrict__ ci,
                  const double* __restrict__ val, const double* __restrict__ h, int n, int count,
                  const int8_t* __restrict__ spins, double* __restrict__ out) {
  // CTA (x, y): replicas 32x .. 32x + 31, sites [y n / Y, (y + 1) n / Y); with
  // Y > 1 the sums go to out[y * count + replica], summed in order of y by
  // energy_sum_kernel (no dependence on timing)
  extern __shared__ uint32_t wsh[];  // [n] words, then [8][32] partial sums
  const int v0 = blockIdx.x * 32;
  const int ilo = (int)(((int64_t)blockIdx.y * n) / gridDim.y);
  const int ihi = (int)(((int64_t)(blockIdx.y + 1) * n) / gridDim.y);
  const int nv = min(32, count - v0);
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    uint32_t w = 0;
    for (int r = 0; r < nv; ++r)
      if (spins[(size_t)(v0 + r) * n + i] < 0) w |= 1u << r;
    wsh[i] = w;
  }
  __syncthreads();
  double acc[32];
#pragma unroll
  for (int r = 0; r < 32; ++r) acc[r] = 0.0;
  for (int i = ilo + threadIdx.x; i < ihi; i += blockDim.x) {
    const uint32_t wi = wsh[i];
    const double hi = h[i];
#pragma unroll
    for (int r = 0; r < 32; ++r) acc[r] += ((wi >> r) & 1u) ? -hi : hi;
    const int p1 = rp[i + 1];
    for (int p = rp[i]; p < p1; ++p) {
      const int j = ci[p];
      if (j <= i) continue;
      const uint32_t x = wi ^ wsh[j];
      const double v = val[p];
#pragma unroll
      for (int r = 0; r < 32; ++r) acc[r] += ((x >> r) & 1u) ? -v : v;
    }
  }
  // warp reduction, then warps in order
  double* part = reinterpret_cast<double*>(wsh + ((n + 1) & ~1));
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
  for (int r = 0; r < 32; ++r) {
    double x = acc[r];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    if (lane == 0) part[warp * 32 + r] = x;
  }
  __syncthreads();
  if (threadIdx.x < nv) {
    double t = 0.0;
    for (int w = 0; w < kEnergyThreads / 32; ++w) t += part[w * 32 + threadIdx.x];
    out[(size_t)blockIdx.y * count + v0 + threadIdx.x] = t;
  }
}

// First slice of minimum energy per replica (get_solution.hpp:69-76, strict <).
__global__ void best_slice_kernel(const double* __restrict__ e, int R, int T, int32_t* __restrict__ best) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= R) return;
  int b = 0;
  double m = e[(size_t)r * T];
  for (int t = 1; t < T; ++t) {
    const double v = e[(size_t)r * T + t];
    if (v < m) {
      m = v;
      b = t;
    }
  }
  best[r] = b;
}

// int8 [R][n] -> words [ceil(R/32)][n]; bit j of word (g, i) set iff replica
// 32g+j has s_i = -1.  Replicas past R read as +1.
__global__ void pack_kernel(const int8_t* __restrict__ spins, int R, int n, uint32_t* __restrict__ words) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int g = blockIdx.y;
  if (i >= n) return;
  uint32_t w = 0;
  for (int j = 0; j < 32; ++j) {
    const int r = 32 * g + j;
    if (r < R && spins[(size_t)r * n + i] < 0) w |= 1u << j;
  }
  words[(size_t)g * n + i] = w;
}

__global__ void unpack_kernel(const uint32_t* __restrict__ words, int R, int n, int8_t* __restrict__ spins) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int g = blockIdx.y;
  if (i >= n) return;
  const uint32_t w = words[(size_t)g * n + i];
  for (int j = 0; j < 32; ++j) {
    const int r = 32 * g + j;
    if (r < R) spins[(size_t)r * n + i] = ((w >> j) & 1u) ? (int8_t)-1 : (int8_t)1;
  }
}

}  // namespace

static cudaError_t colour_build(oj_graph* g) {
  const int n = g->n, ncol = g->info.num_colours;
  std::vector<int32_t> order(g->order), slot(n);
  std::vector<int4> cls(ncol);
  std::vector<int2> site(n), slice;
  std::vector<int2> ent;
  auto deg = [&](int i) { return g->rp[i + 1] - g->rp[i]; };
  auto plan = std::make_unique<ColourPlan>();
  plan->ncol = ncol;
  for (int c = 0; c < ncol; ++c) {
    std::stable_sort(order.begin() + g->coff[c], order.begin() + g->coff[c + 1],
                     [&](int x, int y) { return deg(x) > deg(y); });
    plan->max_class = std::max(plan->max_class, g->coff[c + 1] - g->coff[c]);
  }
  for (int s = 0; s < n; ++s) {
    slot[order[s]] = s;
    int hb;
    std::memcpy(&hb, &g->h[order[s]], 4);
    site[s] = make_int2(order[s], hb);
  }
  size_t total = 0;
  for (int c = 0; c < ncol; ++c)
    for (int s = g->coff[c]; s < g->coff[c + 1]; s += 32)
      total += (size_t)std::min(32, g->coff[c + 1] - s) * (size_t)deg(order[s]);
  if (total > (size_t)INT32_MAX) return cudaErrorMemoryAllocation;
  ent.assign(std::max<size_t>(total, 1), make_int2(0, 0));
  size_t off = 0;
  for (int c = 0; c < ncol; ++c) {
    cls[c] = make_int4(g->coff[c], g->coff[c + 1] - g->coff[c], (int)slice.size(), 0);
    for (int s = g->coff[c]; s < g->coff[c + 1]; s += 32) {
      const int terms = deg(order[s]);  // the slice's largest degree
      const int width = std::min(32, g->coff[c + 1] - s);
      slice.push_back(make_int2((int)off, terms));
      for (int l = 0; l < width; ++l) {
        const int i = order[s + l];
        for (int p = 0; p < deg(i); ++p) {
          int vb;
          std::memcpy(&vb, &g->val[g->rp[i] + p], 4);
          ent[off + (size_t)width * p + l] = make_int2(slot[g->ci[g->rp[i] + p]], vb);
        }
      }
      off += (size_t)width * terms;
    }
  }
  auto al = [](size_t b) { return (b + 255) & ~(size_t)255; };
  const size_t b_site = al(site.size() * 8 + 8), b_cls = al(cls.size() * 16 + 16), b_slice = al(slice.size() * 8 + 8);
  cudaError_t e = plan->tables.ensure(b_site + b_cls + b_slice + al(ent.size() * 8));
  if (e != cudaSuccess) return e;
  char* base = plan->tables.as<char>();
  plan->site = reinterpret_cast<int2*>(base);
  plan->cls = reinterpret_cast<int4*>(base + b_site);
  plan->slice = reinterpret_cast<int2*>(base + b_site + b_cls);
  plan->ent = reinterpret_cast<int2*>(base + b_site + b_cls + b_slice);
  std::vector<char> host(b_site + b_cls + b_slice + al(ent.size() * 8));
  std::memcpy(host.data(), site.data(), site.size() * 8);
  std::memcpy(host.data() + b_site, cls.data(), cls.size() * 16);
  std::memcpy(host.data() + b_site + b_cls, slice.data(), slice.size() * 8);
  std::memcpy(host.data() + b_site + b_cls + b_slice, ent.data(), ent.size() * 8);
  if ((e = copy_tables(base, host.data(), host.size())) != cudaSuccess) return e;
  g->cplan = std::move(plan);
  return cudaSuccess;
}

// Builds the graph's ColourPlan (once).  No exception leaves it: its callers
// are reached through the C interface.  A host or device allocation that fails
// is reported as out of memory, and so are lists that pad to more entries than
// an int counts; the run then takes the kernels that read the graph's own lists.
cudaError_t colour_prepare(oj_graph* g) {
  const std::lock_guard<std::mutex> lock(g->cplan_lock);
  if (g->cplan) return cudaSuccess;
  try {
    return colour_build(g);
  } catch (...) {
    return cudaErrorMemoryAllocation;
  }
}

namespace {

ColourArgs colour_args(const oj_graph* g, int R, int T, int8_t* spins, int64_t nsweeps, const RngBase& rb) {
  const ColourPlan& pl = *g->cplan;
  ColourArgs a;
  a.site = pl.site;
  a.cls = pl.cls;
  a.slice = pl.slice;
  a.ent = pl.ent;
  a.ncol = pl.ncol;
  a.n = g->n;
  a.R = R;
  a.T = T;
  a.spins = spins;
  a.betas = nullptr;
  a.coef = nullptr;
  a.nsweeps = nsweeps;
  a.keys = ojd::make_keys(rb.k0, rb.k1);
  a.sweep0 = rb.sweep0;
  a.rep0 = rb.rep0;
  a.flips = rb.flips;
  return a;
}

// Threads of a CTA (whole warps): one per item of the largest class, the SM's
// 1024 (64 registers each) shared by the CTAs that run on it together.
int colour_threads(int64_t items, int64_t ctas, int sms) {
  const int64_t share = kColourThreads / std::min<int64_t>(8, std::max<int64_t>(1, (ctas + sms - 1) / sms)) / 32 * 32;
  return (int)std::max<int64_t>(64, std::min((items + 31) / 32 * 32, share));
}

// Long neighbour lists: from a mean degree of 32 on (SQA, 300 sites, complete:
// 14.4 -> 9.3 ms a sweep with 16 entries in flight; the registers cost 5 % on a
// Chimera lattice's lists of 6).
bool colour_long(const oj_graph* g) { return g->info.nnz >= 32 * (int64_t)g->n; }

template <class Kern>
cudaError_t colour_launch(Kern kern, const ColourArgs& a, int ctas, int threads, size_t smem, cudaStream_t st) {
  const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  kern<<<ctas, threads, smem, st>>>(a);
  return cudaGetLastError();
}

}  // namespace

cudaError_t launch_sa_colour(const oj_graph* g, int R, int8_t* spins, const float* betas,
                             int64_t nsweeps, RngBase rb, cudaStream_t st, int* launches) {
  if (seq_applies(g, 1)) return launch_sa_seq(g, R, spins, betas, nsweeps, rb, st, launches);
  if (launches) ++*launches;
  const bool fits = g->n <= kSmemBudget;
  const cudaError_t pe = fits ? colour_prepare(const_cast<oj_graph*>(g)) : cudaSuccess;
  if (!fits || pe == cudaErrorMemoryAllocation) {
    cudaGetLastError();
    sa_colour_global_kernel<<<(R + 3) / 4, kColourGlobalThreads, 0, st>>>(
        g->d_rp.as<int32_t>(), g->d_ci.as<int32_t>(), g->d_val.as<float>(), g->d_h.as<float>(),
        g->d_order.as<int32_t>(), g->d_coff.as<int32_t>(), g->info.num_colours, g->n, R, spins, betas, nsweeps, rb);
    return cudaGetLastError();
  }
  if (pe != cudaSuccess) return pe;
  int sms = 0;
  const cudaError_t e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, g->device);
  if (e != cudaSuccess) return e;
  ColourArgs a = colour_args(g, R, 1, spins, nsweeps, rb);
  a.betas = betas;
  // eight replicas a CTA share the neighbour entries; four where that leaves
  // SMs without work
  const int ctas8 = (R + 7) / 8, ctas4 = (R + 3) / 4;
  const int nq = ctas4 <= sms ? 1 : 2, ctas = nq == 1 ? ctas4 : ctas8;
  const int threads = colour_threads(g->cplan->max_class, ctas, sms);
  const size_t smem = g->n;
  if (colour_long(g))
    return nq == 1 ? colour_launch(sa_colour_kernel<1, true>, a, ctas, threads, smem, st)
                   : colour_launch(sa_colour_kernel<2, true>, a, ctas, threads, smem, st);
  return nq == 1 ? colour_launch(sa_colour_kernel<1, false>, a, ctas, threads, smem, st)
                 : colour_launch(sa_colour_kernel<2, false>, a, ctas, threads, smem, st);
}

cudaError_t launch_sqa_colour(const oj_graph* g, int R, int T, int8_t* spins, const float2* coef,
                              int64_t nsweeps, RngBase rb, cudaStream_t st, int* launches) {
  if (seq_applies(g, T)) return launch_sqa_seq(g, R, T, spins, coef, nsweeps, rb, st, launches);
  if (launches) ++*launches;
  const int octets = (T + 7) / 8;
  const size_t smem = (size_t)octets * g->n;
  const bool fits = smem <= (size_t)kSmemBudget;
  const cudaError_t pe = fits ? colour_prepare(const_cast<oj_graph*>(g)) : cudaSuccess;
  if (!fits || pe == cudaErrorMemoryAllocation) {
    cudaGetLastError();
    sqa_colour_global_kernel<<<R, kSqaGlobalThreads, 0, st>>>(
        g->d_rp.as<int32_t>(), g->d_ci.as<int32_t>(), g->d_val.as<float>(), g->d_h.as<float>(),
        g->d_order.as<int32_t>(), g->d_coff.as<int32_t>(), g->info.num_colours, g->n, T, spins, coef, nsweeps, rb);
    return cudaGetLastError();
  }
  if (pe != cudaSuccess) return pe;
  int sms = 0;
  const cudaError_t e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, g->device);
  if (e != cudaSuccess) return e;
  ColourArgs a = colour_args(g, R, T, spins, nsweeps, rb);
  a.coef = coef;
  const int threads = colour_threads((int64_t)octets * ((g->cplan->max_class + 31) / 32 * 32), R, sms);
  const bool lg = colour_long(g);
  if (T <= 2)
    return lg ? colour_launch(sqa_colour_kernel<1, true>, a, R, threads, smem, st)
              : colour_launch(sqa_colour_kernel<1, false>, a, R, threads, smem, st);
  if (T <= 4)
    return lg ? colour_launch(sqa_colour_kernel<2, true>, a, R, threads, smem, st)
              : colour_launch(sqa_colour_kernel<2, false>, a, R, threads, smem, st);
  return lg ? colour_launch(sqa_colour_kernel<4, true>, a, R, threads, smem, st)
            : colour_launch(sqa_colour_kernel<4, false>, a, R, threads, smem, st);
}

// out[v] = sum over y of parts[y * count + v], y in order.
__global__ void energy_sum_kernel(const double* __restrict__ parts, int nsplit, int count, double* __restrict__ out) {
  const int v = blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= count) return;
  double t = 0.0;
  for (int y = 0; y < nsplit; ++y) t += parts[(size_t)y * count + v];
  out[v] = t;
}

int energy_splits(const oj_graph* g, int count, int sm_count) {
  // sites split over CTAs until the grid covers the SMs twice (at least 256
  // sites a CTA)
  const int groups = (count + 31) / 32;
  int k = 1;
  while (k < 16 && groups * k < 2 * sm_count && g->n / (2 * k) >= 256) k *= 2;
  return k;
}

cudaError_t launch_energy(const oj_graph* g, int count, const int8_t* spins, double* out, cudaStream_t st,
                          int nsplit, double* parts) {
  if (count <= 0) return cudaSuccess;
  if (nsplit < 1 || (nsplit > 1 && !parts)) return cudaErrorInvalidValue;
  const size_t smem = (size_t)((g->n + 1) & ~1) * 4 + (kEnergyThreads / 32) * 32 * 8;
  auto kern = energy_kernel;
  if (smem > 48 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
  }
  kern<<<dim3((count + 31) / 32, nsplit), kEnergyThreads, smem, st>>>(
      g->d_rp.as<int32_t>(), g->d_ci.as<int32_t>(), g->d_val64.as<double>(), g->d_h64.as<double>(), g->n, count,
      spins, nsplit > 1 ? parts : out);
  if (nsplit > 1) {
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    energy_sum_kernel<<<(count + 255) / 256, 256, 0, st>>>(parts, nsplit, count, out);
  }
  return cudaGetLastError();
}

cudaError_t launch_best_slice(const double* energies, int R, int T, int32_t* best, cudaStream_t st) {
  best_slice_kernel<<<(R + 127) / 128, 128, 0, st>>>(energies, R, T, best);
  return cudaGetLastError();
}

cudaError_t launch_pack(const int8_t* spins, int R, int n, uint32_t* words, cudaStream_t st) {
  dim3 grid((n + 255) / 256, (R + 31) / 32);
  pack_kernel<<<grid, 256, 0, st>>>(spins, R, n, words);
  return cudaGetLastError();
}

cudaError_t launch_unpack(const uint32_t* words, int R, int n, int8_t* spins, cudaStream_t st) {
  dim3 grid((n + 255) / 256, (R + 31) / 32);
  unpack_kernel<<<grid, 256, 0, st>>>(words, R, n, spins);
  return cudaGetLastError();
}

cudaError_t pack_preload() {
  cudaFuncAttributes fa;
  cudaError_t e = cudaFuncGetAttributes(&fa, pack_kernel);
  return e != cudaSuccess ? e : cudaFuncGetAttributes(&fa, unpack_kernel);
}

}  // namespace oj

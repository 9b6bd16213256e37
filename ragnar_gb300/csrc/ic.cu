// Inverse-Compton spectrum on sm_103a: ICSpectrum (ic.cpp:15-46), ic::Kernel
// (ic.hpp:67-94) and KNfunc (ic.hpp:20-25).
//
//   S[e] = sum_g sum_s f_g (f_s / e_s) e^2 KN(Gamma, q) / g^k      (k = 1 for log-spaced
//          gamma bins, 2 for linear ones), over the (g, s) pairs with e <= g Gamma / (1 + Gamma),
//   Gamma = 4 g e_s,  q = (e / g) / (Gamma (1 - e / g)),
//   KN(Gamma, q) = 2 q ln q + (1 - q) (1 + 2 q + (Gamma q)^2 / (2 (1 + Gamma q))).
//
// Rewritten so that what depends on (e, g) and what depends on the soft photon separate:
//   t = Gamma q = e / (g - e),  z = t / g,  q = z i_s with i_s = 1 / (4 e_s),
//   e <= g Gamma / (1 + Gamma)  <=>  q <= 1 (e < g),  h = t^2 / (2 (1 + t)),
//   KN = (1 + h) + (1 - h) q - 2 q^2 + 2 q ln q.
//
// Regular soft photons (up to 16384 in any order or any number in ascending order, valid
// energies in [1e-30, 1e30] and |w_s| <= 1e30, w_s = f_s / e_s: every tabulated distribution).
// In descending order of i_s the photons with q <= 1 are a suffix s >= j of the table, and
// with q_j = z i_j, the largest q of the suffix,
//   sum_{s >= j} w_s KN = W0 + q V1 - 2 q^2 V2 + 2 q (V1 ln q + V3) + h (W0 - q V1),  q = q_j,
//   W0 = sum w,  V1 = sum w r,  V2 = sum w r^2,  V3 = sum w r ln r,  r = i_s / i_j in (0, 1],
// so one (gamma bin, IC bin) pair costs a binary search for j and a fixed number of
// operations instead of a logarithm per soft photon: the work is ng x ne log2(ns), not
// ng x ne x ns.  The suffix sums are formed in FP64 and stored as double-floats, and the
// pair's terms are summed in double-float arithmetic: near q = 1 they cancel to
// KN ~ (1 + h)(1 - q), which FP32 sums would leave with an error of 1e-7 / (1 - q).  FP32
// pipes do it at about seven times the FP64 pipe's rate here (1.6 FP64 operations per clock
// and SM against ~110 FP32).
//
// Any other soft photons (infinities and NaN among them) take the direct kernel, with L = 2 ln 2 and p = L q
// (2 q ln q = p (log2 p - log2 L)):
//   KN = p log2 p + ((1 + h) + ((1 - h) / L - log2 L) p - (2 / L^2) p^2),
// per eval FMUL (p), MUFU.LG2, two FFMA (quadratic), FFMA (log term), max(KN, 0), FFMA into the
// FP32 accumulator.  max(KN, 0) is KN [q <= 1]: at fixed h, KN(1) = 0, KN'(1) = -1 - h < 0 and
// KN'' = 2/q - 4 < 0 for q > 1/2, so KN < 0 for every q > 1, while KN >= 0 on (0, 1] (the
// Klein-Nishina kernel).  Evals with p = inf (masked soft photons; (e, g) pairs that no soft
// photon reaches, e >= g or an invalid e, which get pg = inf) evaluate to NaN, which max(., 0)
// also maps to 0.  q >= 1e-30 is guaranteed by a floor on t/g set per (e, g) from the smallest
// 1 / (4 e_s), so the log's argument is a normal float or inf.  Lanes own IC bins (K rows of 32
// per lane, 512-bin slices in blockIdx.y); warps take (gamma bin, 64-soft-photon chunk) items;
// per item the FP32 sums are scaled by e^2 f_g / g^k and folded into a double-float.
//
// Which of the two runs is decided on the device (ic_sums_kernel), so a call needs no
// host synchronisation; the other kernel's blocks return at once.  Both sum their warps in
// FP64 at a block's end into one partial row, and the rows are summed in a fixed order
// (deterministic).  Non-positive or non-finite IC bins give 0 (the reference produces NaN
// there).
//
// Measured at 1024 gamma x 1024 soft-photon x 1024 IC bins, back to back on one stream: 47.5 us a
// call (52 us with the photons shuffled) against 369 us with every triple evaluated, the largest
// error against FP64 1e-7 against 2.2e-5 (a line of photons at the Klein-Nishina edge).  The
// kernels: terms 8 us, sums 9.5 us (FP64 pipe of four SMs), pairs 23 us (issue and latency: ~340
// instructions a pair), the direct kernel's early return 4 us, reduction 5 us (under a profiler,
// serialised).
#include "moments_common.cuh"

#include <algorithm>
#include <cmath>

namespace rg {

  namespace {

    constexpr int kIcThreads = 256;
    constexpr int kIcWarps   = kIcThreads / 32;
    constexpr int kIcSlice   = 512; // the widest slice of IC bins (K = 16 rows of 32 per lane)
    constexpr int kIcSChunk  = 64; // soft photons per work item
    constexpr int kIcMaxRows = 16; // rows of 32 IC bins per lane (the slice width is rows x 32)

    // Suffix sums of a regular soft-photon table, as double-floats (hi, lo) per photon.
    struct IcSums {
      float2* i4; // 1 / (4 e_s)
      float2* w0; // W0
      float2* v1; // V1, V2, V3 relative to the photon's own 1 / (4 e_s)
      float2* v2;
      float2* v3;
    };

    struct IcParams {
      const float* gb;      // ng gamma (gamma beta) bins
      const float* fp;      // ng particle distribution
      int          ng;
      int          log_spaced;
      const float* es;      // ns soft-photon energies and distribution, as given
      const float* fs;
      float*       inv4es;  // ns, in the order of the sums: 1 / (4 e_s), inf for masked photons
      float*       inv4es_min; // min over s of 1 / (4 e_s) (positive values), one float
      float*       ws;      // ns: f_s / e_s
      double*      terms;   // [6][ns]: w, w i, w i^2, w i ln i, ln i, 1 / i with i = 1 / (4 e_s)
      float2*      blocks;  // per block of ic_terms_kernel: smallest i (as inv4es_min), 1 if its photons are in order and in range
      int          nblocks;
      double*      tiles;   // [4][ntiles]: sums of the first four terms over a tile of kTile photons (more than one tile)
      int          ntiles;
      int*         regular; // 1: the pair kernel runs, 0: the direct kernel
      IcSums       sums;
      int          ns;
      const float* eic;     // ne IC photon energies
      int          ne;
      int          nslices; // direct kernel: slices of slice_w IC bins (K x 32)
      int          slice_w;
      double*      partials;  // direct kernel: [grid][nslices][slice_w], one row per block
      double*      pairs;     // pair kernel: [splits][ne], one row per range of gamma bins
    };

    // ---- soft-photon tables ---------------------------------------------------------------

    constexpr int kPrepThreads = 256;
    constexpr int kPrepItems   = 4; // photons per thread and tile
    constexpr int kTile        = kPrepThreads * kPrepItems;
    constexpr int kRankMax     = 16384; // photons that are ranked when they are out of order
    constexpr int kRankTile    = 1024; // a multiple of a block's photons
    constexpr int kRankWays    = 4;     // threads that share a photon's comparisons
    // energies and largest |weight| of a regular table: far enough from the ends of the float range for
    // every double-float product of the pair kernel.  Small weights need no bound: their products lose
    // low parts below 2^-126, but no more than the direct kernel's FP32 loses there (weights of 1e-38:
    // 1.1e-7 against 3.2e-7).
    constexpr float kRegularLo = 1e-30f, kRegularHi = 1e30f;

    __device__ __forceinline__ ff ff_div(ff a, ff b) {
      const float r  = __frcp_rn(b.hi);
      const float q0 = __fmul_rn(a.hi, r);
      const float e  = __fadd_rn(__fmaf_rn(-q0, b.hi, a.hi), __fmaf_rn(-q0, b.lo, a.lo));
      return fast_two_sum(q0, __fmul_rn(e, r));
    }

    __device__ __forceinline__ double ff_to_double(ff a) {
      return static_cast<double>(a.hi) + static_cast<double>(a.lo);
    }

    __device__ __forceinline__ float2 double_to_ff(double d) {
      const float h = __double2float_rn(d);
      return make_float2(h, isfinite(h) ? __double2float_rn(d - static_cast<double>(h)) : 0.0f);
    }

    // 1 / (4 e) of a valid photon energy, inf for one that contributes nothing (e <= 0, not
    // finite, or 1 / (4 e) above the float range): masked photons come first in the order.
    __device__ __forceinline__ float ic_inv4(float e) {
      return (e > 0.0f && isfinite(e)) ? __frcp_rn(__fmul_rn(4.0f, e)) : __int_as_float(0x7f800000);
    }

    // Of photons without a positive 1 / (4 e_s): above any such value of a positive float.
    __device__ __forceinline__ float no_min() {
      return __int_as_float(0x7f7f7f7f);
    }

    // v's smallest value over the block, in thread 0
    __device__ __forceinline__ float block_min(float v) {
      __shared__ float wmin[kPrepThreads / 32];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        v = fminf(v, __shfl_xor_sync(0xffffffffu, v, o));
      }
      if ((threadIdx.x & 31) == 0) {
        wmin[threadIdx.x >> 5] = v;
      }
      __syncthreads();
      if (threadIdx.x == 0) {
        for (int w = 1; w < kPrepThreads / 32; ++w) {
          v = fminf(v, wmin[w]);
        }
      }
      return v;
    }

    // v's sum over the block (in a fixed order), the same in every thread
    __device__ __forceinline__ double block_sum(double v) {
      __shared__ double wsum[kPrepThreads / 32];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        v += __shfl_xor_sync(0xffffffffu, v, o);
      }
      __syncthreads(); // the last sum's values are read
      if ((threadIdx.x & 31) == 0) {
        wsum[threadIdx.x >> 5] = v;
      }
      __syncthreads();
      v = 0.0;
#pragma unroll
      for (int w = 0; w < kPrepThreads / 32; ++w) {
        v += wsum[w];
      }
      return v;
    }

    // Per photon: its place in descending order of 1 / (4 e_s), and its terms of the four sums.  A table
    // already in order keeps its places; one of up to kRankMax photons in any other order is ranked by
    // comparing all pairs (ns^2 comparisons against ng x ne x ns evals of the direct kernel); a longer
    // one is left to the direct kernel.  Where ranks may be needed, kRankWays threads share a
    // photon's comparisons (and a block has fewer photons), so that they fill the chip: 16384 photons
    // out of order take 56 us more than in order, with a thread per photon 215 us.  Quotients and
    // logarithms are taken in double-floats, as FP64 issues at 1.6 operations per clock and SM.
    __global__ void __launch_bounds__(kPrepThreads) ic_terms_kernel(const __grid_constant__ IcParams p) {
      __shared__ float4 keys[kRankTile / 4];
      const bool rank = p.ns <= kRankMax;
      const int  ways = rank ? kRankWays : 1, part = threadIdx.x & (ways - 1);
      const int  s0   = blockIdx.x * (kPrepThreads / ways), s = s0 + static_cast<int>(threadIdx.x) / ways;
      const bool mine = s < p.ns && part == 0;
      // in order over the whole table (each block decides for itself) or, above kRankMax, over
      // this block's photons
      bool out_of_order = false;
      if (rank) {
#pragma unroll 4
        for (int k = threadIdx.x; k < p.ns - 1; k += kPrepThreads) {
          out_of_order = out_of_order || ic_inv4(p.es[k]) < ic_inv4(p.es[k + 1]);
        }
      } else {
        out_of_order = s < p.ns - 1 && ic_inv4(p.es[s]) < ic_inv4(p.es[s + 1]);
      }
      const bool  unsorted = __syncthreads_or(out_of_order) != 0;
      const float e = s < p.ns ? p.es[s] : 0.0f, f = s < p.ns ? p.fs[s] : 0.0f;
      const float i4  = ic_inv4(e);
      const bool  use = i4 <= 3.402823466e38f; // false for inf: a photon that contributes nothing
      int         at  = s;
      if (unsorted && rank) {
        at = 0;
        for (int t0 = 0; t0 < p.ns; t0 += kRankTile) {
          __syncthreads();
          for (int k = threadIdx.x; k < kRankTile; k += kPrepThreads) {
            reinterpret_cast<float*>(keys)[k] = t0 + k < p.ns ? ic_inv4(p.es[t0 + k]) : -1.0f; // before no photon
          }
          __syncthreads();
          // equal keys keep their order: photons before this one count where they are equal too
          const bool before = t0 + kRankTile <= s0, after = t0 > s0;
#pragma unroll 4
          for (int k = part; k < kRankTile / 4; k += kRankWays) {
            const float4 v = keys[k];
            if (before) {
              at += (v.x >= i4) + (v.y >= i4) + (v.z >= i4) + (v.w >= i4);
            } else if (after) {
              at += (v.x > i4) + (v.y > i4) + (v.z > i4) + (v.w > i4);
            } else {
              const int t = t0 + 4 * k;
              at += (v.x > i4 || (v.x == i4 && t < s)) + (v.y > i4 || (v.y == i4 && t + 1 < s)) +
                    (v.z > i4 || (v.z == i4 && t + 2 < s)) + (v.w > i4 || (v.w == i4 && t + 3 < s));
            }
          }
        }
#pragma unroll
        for (int o = 1; o < kRankWays; o <<= 1) {
          at += __shfl_xor_sync(0xffffffffu, at, o);
        }
      }
      bool ok = rank || !unsorted;
      if (mine) {
        const float wf = use ? __fdiv_rn(f, e) : 0.0f;
        p.inv4es[at]   = i4;
        p.ws[at]       = wf;
        ok = ok && (!use || (e >= kRegularLo && e <= kRegularHi && fabsf(wf) <= kRegularHi));
        double w = 0.0, i = 0.0, lni = 0.0, ri = 0.0;
        ff     iv { i4, 0.0f };
        if (use) {
          iv              = ff_div(ff { 0.25f, 0.0f }, ff { e, 0.0f });
          w               = ff_to_double(ff_div(ff { f, 0.0f }, ff { e, 0.0f }));
          i               = ff_to_double(iv);
          ri              = 4.0 * static_cast<double>(e);
          const LnParts l = ln_parts(ff { e, 0.0f }); // ln i = -ln(4 e)
          lni             = -((static_cast<double>(l.e) + 2.0) * M_LN2 + ff_to_double(ff { l.h, l.l }));
        }
        const double  wi = w * i;
        const int64_t ns = p.ns; // 6 ns entries: more than 2^31 from 3.6e8 photons
        p.sums.i4[at]        = make_float2(iv.hi, iv.lo);
        p.terms[at]          = w;
        p.terms[ns + at]     = wi;
        p.terms[2 * ns + at] = wi * i;
        p.terms[3 * ns + at] = wi * lni;
        p.terms[4 * ns + at] = lni;
        p.terms[5 * ns + at] = ri;
      }
      const int all  = __syncthreads_and(ok);
      float     imin = mine && i4 > 0.0f ? fminf(i4, no_min()) : no_min();
      imin           = block_min(imin);
      if (threadIdx.x == 0) {
        p.blocks[blockIdx.x] = make_float2(imin, all ? 1.0f : 0.0f);
        if (!all && p.ns > kRankMax) {
          *p.regular = 0; // set before the launch: long tables skip their sums
        }
      }
    }

    // The sum of a term (0 .. 3) over a tile, for the tiles before it: block 4 tile + term.
    __global__ void __launch_bounds__(kPrepThreads) ic_tiles_kernel(const __grid_constant__ IcParams p) {
      const int     which = blockIdx.x & 3, tile = blockIdx.x >> 2;
      const int64_t base = static_cast<int64_t>(tile) * kTile;
      if (p.ns > kRankMax && !*p.regular) {
        return;
      }
      double        v    = 0.0;
#pragma unroll
      for (int k = 0; k < kPrepItems; ++k) {
        const int64_t s = base + k * kPrepThreads + threadIdx.x;
        v += s < p.ns ? p.terms[which * static_cast<int64_t>(p.ns) + s] : 0.0;
      }
      v = block_sum(v);
      if (threadIdx.x == 0) {
        p.tiles[static_cast<int64_t>(which) * p.ntiles + tile] = v;
      }
    }

    // One block per sum (0: W0, 1: V1, 2: V2, 3: V3) and tile of photons (block 4 tile + sum), a
    // thread summing four consecutive ones from the tile's end, in FP64 (the sums' range exceeds
    // FP32's), after the sums of the later tiles; several SMs share the FP64 additions.  Block 0
    // also decides which kernel runs.  10 gamma bins x 10 IC bins: 16384 photons 62 us (one block walking
    // all tiles, 7 us each: 160), 1e5 62 (720), 1e6 0.26 ms (7.1); evaluated directly 40, 59 and 0.27 ms.
    __global__ void __launch_bounds__(kPrepThreads) ic_sums_kernel(const __grid_constant__ IcParams p) {
      __shared__ double wtot[2][kPrepThreads / 32];
      const int     which = blockIdx.x & 3, tile = blockIdx.x >> 2, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
      const int64_t ns   = p.ns, first = static_cast<int64_t>(tile) * kTile, end = min(ns, first + kTile);
      double        carry = 0.0, carry1 = 0.0; // sums over the later tiles (carry1: V3's sum of w i)
      if (p.ns > kRankMax && blockIdx.x != 0 && !*p.regular) {
        return;
      }
      if (p.ntiles > 1) {
        const double* later = p.tiles + static_cast<int64_t>(which) * p.ntiles;
        const double* later1 = p.tiles + p.ntiles;
        for (int k = tile + 1 + tid; k < p.ntiles; k += kPrepThreads) {
          carry += later[k];
          carry1 += which == 3 ? later1[k] : 0.0;
        }
        carry  = block_sum(carry);
        carry1 = which == 3 ? block_sum(carry1) : 0.0;
      }
      double a[kPrepItems], a1[kPrepItems];
      double t = 0.0, t1 = 0.0;
#pragma unroll
      for (int k = 0; k < kPrepItems; ++k) {
        const int64_t s = end - 1 - (tid * kPrepItems + k);
        const bool    in = s >= first;
        a[k]  = in ? p.terms[which * ns + s] : 0.0;
        a1[k] = (in && which == 3) ? p.terms[ns + s] : 0.0;
        t += a[k];
        t1 += a1[k];
      }
      // inclusive sums over the warp's threads
      double x = t, x1 = t1;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const double y  = __shfl_up_sync(0xffffffffu, x, o);
        const double y1 = which == 3 ? __shfl_up_sync(0xffffffffu, x1, o) : 0.0;
        if (lane >= o) {
          x += y;
          x1 += y1;
        }
      }
      if (lane == 31) {
        wtot[0][warp] = x;
        wtot[1][warp] = x1;
      }
      __syncthreads();
      for (int w = 0; w < warp; ++w) {
        carry += wtot[0][w];
        carry1 += wtot[1][w];
      }
      // the lane below holds this lane's exclusive sum within the warp
      const double up = __shfl_up_sync(0xffffffffu, x, 1), up1 = __shfl_up_sync(0xffffffffu, x1, 1);
      double       run = lane > 0 ? carry + up : carry, run1 = lane > 0 ? carry1 + up1 : carry1;
#pragma unroll
      for (int k = 0; k < kPrepItems; ++k) {
        const int64_t s = end - 1 - (tid * kPrepItems + k);
        run += a[k];
        run1 += a1[k];
        if (s >= first) {
          if (which == 0) {
            p.sums.w0[s] = double_to_ff(run);
          } else {
            const double ri = p.terms[5 * ns + s];
            if (which == 1) {
              p.sums.v1[s] = double_to_ff(run * ri);
            } else if (which == 2) {
              p.sums.v2[s] = double_to_ff(run * ri * ri);
            } else {
              p.sums.v3[s] = double_to_ff((run - p.terms[4 * ns + s] * run1) * ri);
            }
          }
        }
      }
      if (blockIdx.x == 0) {
        bool  ok   = true;
        float imin = no_min();
        for (int k = tid; k < p.nblocks; k += kPrepThreads) {
          const float2 b = p.blocks[k];
          imin           = fminf(imin, b.x);
          ok             = ok && b.y != 0.0f;
        }
        const int all = __syncthreads_and(ok);
        imin          = block_min(imin);
        if (tid == 0) {
          *p.inv4es_min = imin;
          if (ns <= kRankMax) { // otherwise ic_terms_kernel has said so, and other blocks read it
            *p.regular = all;
          }
        }
      }
    }

    // L = 2 ln 2 rounded to FP32; log2 L and -2 / L^2 of that FP32 value
    constexpr float kIcL     = 1.3862943649291992f;
    constexpr float kIcLog2L = 0.47123363101939075f;

    // What an (IC bin, gamma bin) pair contributes to every eval: pg = L t / g (p = pg / (4 e_s)),
    // 1 + h, and the linear coefficient (1 - h) / L - log2 L; pg = inf for a pair that no soft
    // photon reaches (e >= g or an invalid e).  e: the bin's energy, 0 if invalid.
    __device__ __forceinline__ float4 ic_pair_setup(float e, float gv, float inv_g, float tg_floor) {
      const float d     = __fsub_rn(gv, e);
      const bool  reach = e > 0.0f && d > 0.0f;
      float       t = 0.0f, h = 0.0f;
      if (reach) {
        t = __fdiv_rn(e, d);
        h = __fdiv_rn(__fmul_rn(0.5f, __fmul_rn(t, t)), __fadd_rn(1.0f, t));
      }
      const float pg = reach ? __fmul_rn(kIcL, fmaxf(__fmul_rn(t, inv_g), tg_floor)) : __int_as_float(0x7f800000);
      return make_float4(pg, __fadd_rn(1.0f, h), __fsub_rn(__fdiv_rn(__fsub_rn(1.0f, h), kIcL), kIcLog2L), 0.0f);
    }

    __device__ __forceinline__ float ic_bin_energy(const IcParams& p, int bin) {
      const float e = bin < p.ne ? __ldg(p.eic + bin) : 0.0f;
      return (e > 0.0f && isfinite(e)) ? e : 0.0f;
    }

    // t/g >= this keeps q = (t/g) / (4 e_s) >= 1e-30 for every soft photon with e_s > 0: the
    // log's argument stays a normal float without a per-eval clamp
    __device__ __forceinline__ float ic_tg_floor(const IcParams& p) {
      return __fdiv_rn(1e-30f, *p.inv4es_min);
    }

    // ---- regular soft photons: one (gamma bin, IC bin) pair per thread and step ---------------

    // Lanes own IC bins, warps take gamma bins (every kIcWarps x gridDim.y-th one).
    __global__ void __launch_bounds__(kIcThreads) ic_pair_kernel(const __grid_constant__ IcParams p) {
      __shared__ double red[kIcWarps][32];
      const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
      if (!*p.regular) {
        return;
      }
      const int   bin = blockIdx.x * 32 + lane;
      const float e   = ic_bin_energy(p, bin);
      const float ee  = __fmul_rn(e, e);
      float       hi = 0.0f, lo = 0.0f;
      for (int g = blockIdx.y * kIcWarps + warp; g < p.ng; g += kIcWarps * gridDim.y) {
        const float gv = __ldg(p.gb + g), fv = __ldg(p.fp + g);
        if (!(gv > 0.0f) || !isfinite(gv)) {
          continue; // non-positive or non-finite gamma bins contribute nothing (warp-uniform)
        }
        ff S { 0.0f, 0.0f };
        if (e > 0.0f && gv > e) {
          const ff    t  = ff_div(ff { e, 0.0f }, two_sum(gv, -e));
          const ff    z  = ff_div(t, ff { gv, 0.0f });
          const float h  = __fdiv_rn(__fmul_rn(0.5f * t.hi, t.hi), __fadd_rn(1.0f, t.hi));
          // the first photon with q <= 1 (1 / (4 e_s) descends)
          int j = 0, n = p.ns;
          while (j < n) {
            const int mid = j + ((n - j) >> 1);
            if (__fmul_rn(z.hi, __ldg(p.inv4es + mid)) <= 1.0f) {
              n = mid;
            } else {
              j = mid + 1;
            }
          }
          ff q { 0.0f, 0.0f };
          for (; j < p.ns; ++j) { // q in double-float: the float product may have rounded down to 1
            const float2 iv = __ldg(p.sums.i4 + j);
            q               = ff_mul(z, ff { iv.x, iv.y });
            if (q.hi < 1.0f || (q.hi == 1.0f && q.lo <= 0.0f)) {
              break;
            }
          }
          if (j < p.ns) {
            const float2 w0 = __ldg(p.sums.w0 + j), v1 = __ldg(p.sums.v1 + j);
            const float2 v2 = __ldg(p.sums.v2 + j), v3 = __ldg(p.sums.v3 + j);
            const ff     W0 { w0.x, w0.y }, V1 { v1.x, v1.y }, V2 { v2.x, v2.y }, V3 { v3.x, v3.y };
            S               = W0;
            if (q.hi >= 1e-30f) { // below, KN = 1 + h to rounding
              const LnParts l  = ln_parts_rcp(q);
              const float   fe = static_cast<float>(l.e);
              // e ln2 with ln2 = 0.693145751953125 (16 bits: exact product) + 1.42860677e-6
              ff ln  = two_sum(__fmul_rn(fe, 0.693145751953125f), l.h);
              ln     = fast_two_sum(ln.hi, __fadd_rn(ln.lo, __fmaf_rn(fe, 1.4286068203094173e-6f, l.l)));
              ff c   = ff_add(ff_mul(ln, V1), V3);
              c      = ff_add(c, ff_neg(ff_mul(q, V2)));     // V1 ln q + V3 - q V2
              c      = ff { 2.0f * c.hi, 2.0f * c.lo };
              S      = ff_add(W0, ff_mul(q, ff_add(V1, c)));  // W0 + q V1 + 2 q (...)
            }
            const ff d = ff_add(W0, ff_neg(ff_mul(q, V1)));
            S          = ff_add(S, ff_mul(ff { h, 0.0f }, d));
          }
        }
        // times f_g / g^k and e^2, into the double-float sum
        const float inv_g = __frcp_rn(gv);
        const float fg    = p.log_spaced ? __fmul_rn(fv, inv_g) : __fmul_rn(__fmul_rn(fv, inv_g), inv_g);
        const ff    term  = ff_mul(ff_mul(S, ff { fg, 0.0f }), ff { ee, 0.0f });
        const ff    sm    = two_sum(hi, term.hi);
        hi                = sm.hi;
        lo                = __fadd_rn(lo, __fadd_rn(sm.lo, term.lo));
      }
      red[warp][lane] = static_cast<double>(hi) + static_cast<double>(lo);
      __syncthreads();
      if (warp == 0 && bin < p.ne) {
        double t = 0.0;
#pragma unroll
        for (int w = 0; w < kIcWarps; ++w) {
          t += red[w][lane];
        }
        p.pairs[static_cast<int64_t>(blockIdx.y) * p.ne + bin] = t;
      }
    }

    // ---- any soft photons: every (gamma bin, soft photon, IC bin) evaluated --------------------

    template <int K>
    __global__ void __launch_bounds__(kIcThreads, 2) ic_kernel(const __grid_constant__ IcParams p) {
      if (*p.regular) {
        return;
      }
      const int     lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
      const int     slice = blockIdx.y;
      const int     nsc   = (p.ns + kIcSChunk - 1) / kIcSChunk;
      const int64_t items = static_cast<int64_t>(p.ng) * nsc;
      const int64_t G = gridDim.x, b = blockIdx.x;
      const int64_t i0 = b * items / G, i1 = (b + 1) * items / G;

      // this lane's IC energy of row k (0 for padding and for invalid bins); reloaded
      // where needed (per item) instead of held in registers
      auto energy = [&](int k) -> float { return ic_bin_energy(p, slice * (K * 32) + k * 32 + lane); };
      float hi[K], lo[K];
#pragma unroll
      for (int k = 0; k < K; ++k) {
        hi[k] = 0.0f;
        lo[k] = 0.0f;
      }
      const float kC2      = -1.0406844847835448f; // -2 / L^2
      const float tg_floor = ic_tg_floor(p);

      // A warp's items are consecutive, so that those of one gamma bin share its setup (ic_pair_setup): set up
      // for every item it took 26 us of 388 (1024 gamma bins x 1024 photons x 1024 IC bins,
      // now 8).
      const int64_t w0 = i0 + (i1 - i0) * warp / kIcWarps, w1 = i0 + (i1 - i0) * (warp + 1) / kIcWarps;
      float         pg[K], A0[K], B1[K];
      int           last_g = -1;
      for (int64_t it = w0; it < w1; ++it) {
        const int   g     = static_cast<int>(it / nsc);
        const int   s0    = static_cast<int>(it - static_cast<int64_t>(g) * nsc) * kIcSChunk;
        const int   s1    = min(p.ns, s0 + kIcSChunk);
        const float gv    = __ldg(p.gb + g);
        const float fv    = __ldg(p.fp + g);
        if (!(gv > 0.0f) || !isfinite(gv)) {
          continue; // non-positive or non-finite gamma bins contribute nothing (warp-uniform)
        }
        const float inv_g = __frcp_rn(gv);
        // per (e, g): pg, 1 + h and the linear coefficient (ic_pair_setup);
        // q = (t / g) / (4 e_s) > 1 marks no contribution
        if (g != last_g) {
#pragma unroll
          for (int k = 0; k < K; ++k) {
            const float4 v = ic_pair_setup(energy(k), gv, inv_g, tg_floor);
            pg[k]  = v.x;
            A0[k]  = v.y;
            B1[k]  = v.z;
          }
          last_g = g;
        }
        float acc[K];
#pragma unroll
        for (int k = 0; k < K; ++k) {
          acc[k] = 0.0f;
        }
        for (int s = s0; s < s1; ++s) {
          const float i4 = __ldg(p.inv4es + s);
          const float w  = __ldg(p.ws + s);
#pragma unroll
          for (int k = 0; k < K; ++k) {
            const float pq = __fmul_rn(pg[k], i4);
            // p >= L 1e-30 by the floor on t/g, so the log's argument is a normal float or
            // inf; max(KN, 0) is KN [q <= 1] and maps NaN to 0
            const float lp   = lg2_normal(pq);
            const float poly = __fmaf_rn(__fmaf_rn(kC2, pq, B1[k]), pq, A0[k]);
            const float kn   = __fmaf_rn(pq, lp, poly);
            acc[k]           = __fmaf_rn(w, fmaxf(kn, 0.0f), acc[k]);
          }
        }
        // scale by e^2 f_g / g^k and fold into the double-float sums
        const float fg = p.log_spaced ? __fmul_rn(fv, inv_g) : __fmul_rn(__fmul_rn(fv, inv_g), inv_g);
#pragma unroll
        for (int k = 0; k < K; ++k) {
          const float e    = energy(k);
          const float term = __fmul_rn(__fmul_rn(acc[k], fg), __fmul_rn(e, e));
          const ff    sm   = two_sum(hi[k], term);
          hi[k]            = sm.hi;
          lo[k]            = __fadd_rn(lo[k], sm.lo);
        }
      }
      // the block's warps summed in FP64 in warp order: one partial row per block
      __shared__ double red[kIcWarps * kIcSlice];
#pragma unroll
      for (int k = 0; k < K; ++k) {
        red[warp * (K * 32) + k * 32 + lane] = static_cast<double>(hi[k]) + static_cast<double>(lo[k]);
      }
      __syncthreads();
      double* dst = p.partials + (b * p.nslices + slice) * (K * 32);
      for (int j = threadIdx.x; j < K * 32; j += kIcThreads) {
        double t = 0.0;
#pragma unroll
        for (int w = 0; w < kIcWarps; ++w) {
          t += red[w * (K * 32) + j];
        }
        dst[j] = t;
      }
    }

    // out[e] = sum (fixed order) over the partial rows of the kernel that ran: `splits` rows of
    // ne bins (pair kernel) or `grid` rows of slices (direct kernel); 32 bins x 32 row groups.
    __global__ void __launch_bounds__(1024)
      ic_reduce_kernel(const __grid_constant__ IcParams p, int splits, int grid, float* __restrict__ out) {
      __shared__ double part[32][33];
      const int bin = blockIdx.x * 32 + threadIdx.x, ty = threadIdx.y;
      double    sum = 0.0;
      if (bin < p.ne) {
        const bool    pairs = *p.regular != 0;
        const int     rows  = pairs ? splits : grid;
        const double* src   = pairs ? p.pairs + bin
                                    : p.partials + static_cast<int64_t>(bin / p.slice_w) * p.slice_w + bin % p.slice_w;
        const int64_t step  = pairs ? p.ne : static_cast<int64_t>(p.nslices) * p.slice_w;
        // unrolled so that several rows' loads are in flight (the adds stay in row order)
#pragma unroll 8
        for (int r = ty; r < rows; r += 32) {
          sum += src[r * step];
        }
      }
      part[ty][threadIdx.x] = sum;
      __syncthreads();
      if (ty == 0 && bin < p.ne) {
        double t = 0.0;
        for (int y = 0; y < 32; ++y) {
          t += part[y][threadIdx.x];
        }
        out[bin] = __double2float_rn(t);
      }
    }

    template <int K>
    cudaError_t launch_ic_k(const IcParams& p, dim3 grid, cudaStream_t s) {
      ic_kernel<K><<<grid, kIcThreads, 0, s>>>(p);
      return cudaGetLastError();
    }

    cudaError_t launch_ic(int K, const IcParams& p, dim3 grid, cudaStream_t s) {
      switch (K) {
#define RG_IC_K(k)                                                                                   \
  case k:                                                                                            \
    return launch_ic_k<k>(p, grid, s);
        RG_IC_K(1) RG_IC_K(2) RG_IC_K(3) RG_IC_K(4) RG_IC_K(5) RG_IC_K(6) RG_IC_K(7) RG_IC_K(8)
        RG_IC_K(9) RG_IC_K(10) RG_IC_K(11) RG_IC_K(12) RG_IC_K(13) RG_IC_K(14) RG_IC_K(15) RG_IC_K(16)
#undef RG_IC_K
        default:
          return cudaErrorInvalidValue;
      }
    }

  } // namespace

} // namespace rg

extern "C" {

int rg_ic_spectrum(const float* gbins, const float* f, int32_t ng, int32_t log_spaced, const float* es,
                   const float* fs, int32_t ns, const float* eic, int32_t ne, float* out, void* stream) {
  rg::NvtxRange nvtx_range("ICSpectrum");
  rg::clear_error();
  if (ng < 0 || ns < 0 || ne < 0 || (ng > 0 && (!gbins || !f)) || (ns > 0 && (!es || !fs)) ||
      (ne > 0 && (!eic || !out))) {
    return rg::set_error(RG_ERR_ARGUMENT, "rg_ic_spectrum: bad arguments");
  }
  auto s = static_cast<cudaStream_t>(stream);
  if (ne == 0) {
    return RG_OK;
  }
  if (ng == 0 || ns == 0) {
    RG_CUDA_TRY(cudaMemsetAsync(out, 0, sizeof(float) * ne, s));
    return RG_OK;
  }
  rg::DeviceContext* ctx = nullptr;
  RG_TRY(rg::context(&ctx));
  const int     K       = std::min(rg::kIcMaxRows, (std::min(ne, rg::kIcSlice) + 31) / 32);
  const int     slice_w = K * 32;
  const int     nslices = (ne + slice_w - 1) / slice_w;
  const int64_t items   = static_cast<int64_t>(ng) * ((ns + rg::kIcSChunk - 1) / rg::kIcSChunk);
  const int     grid    = static_cast<int>(std::max<int64_t>(
    1, std::min<int64_t>(2 * ctx->sms, (items + rg::kIcWarps - 1) / rg::kIcWarps)));
  // ranges of gamma bins of the pair kernel: about four blocks per SM, each warp at least one bin
  const int col_blocks = (ne + 31) / 32;
  const int splits     = std::max(1, std::min((ng + rg::kIcWarps - 1) / rg::kIcWarps,
                                              (4 * ctx->sms + col_blocks - 1) / col_blocks));
  // one stream-ordered scratch allocation: photon arrays, sums, partial rows
  const auto     up       = [](size_t v) { return 256 * ((v + 255) / 256); };
  const size_t   n4 = up(sizeof(float) * ns), n8 = up(sizeof(float2) * ns), n48 = up(sizeof(double) * 6 * ns);
  const int      per_block   = ns <= rg::kRankMax ? rg::kPrepThreads / rg::kRankWays : rg::kPrepThreads;
  const int      term_blocks = (ns - 1) / per_block + 1;
  const size_t   off_sums = 2 * n4, off_terms = off_sums + 5 * n8, off_min = off_terms + n48;
  const int      tiles  = (ns - 1) / rg::kTile + 1;
  const size_t   off_blocks = off_min + 256, off_tiles = off_blocks + up(sizeof(float2) * term_blocks);
  const size_t   off_pairs = off_tiles + up(sizeof(double) * 4 * tiles);
  const size_t   off_part = off_pairs + up(sizeof(double) * static_cast<size_t>(splits) * ne);
  const size_t   bytes    = off_part + sizeof(double) * static_cast<size_t>(grid) * nslices * slice_w;
  unsigned char* buf      = nullptr;
  RG_TRY(rg::scratch_alloc(reinterpret_cast<void**>(&buf), bytes, s));
  rg::IcParams p {};
  p.gb         = gbins;
  p.fp         = f;
  p.ng         = ng;
  p.log_spaced = log_spaced ? 1 : 0;
  p.es         = es;
  p.fs         = fs;
  p.inv4es     = reinterpret_cast<float*>(buf);
  p.ws         = reinterpret_cast<float*>(buf + n4);
  float2** sums[5] = { &p.sums.i4, &p.sums.w0, &p.sums.v1, &p.sums.v2, &p.sums.v3 };
  for (int k = 0; k < 5; ++k) {
    *sums[k] = reinterpret_cast<float2*>(buf + off_sums + k * n8);
  }
  p.terms      = reinterpret_cast<double*>(buf + off_terms);
  p.blocks     = reinterpret_cast<float2*>(buf + off_blocks);
  p.nblocks    = term_blocks;
  p.tiles      = reinterpret_cast<double*>(buf + off_tiles);
  p.ntiles     = tiles;
  p.inv4es_min = reinterpret_cast<float*>(buf + off_min);
  p.regular    = reinterpret_cast<int*>(buf + off_min + 128);
  p.ns         = ns;
  p.eic        = eic;
  p.ne         = ne;
  p.nslices    = nslices;
  p.slice_w    = slice_w;
  p.pairs      = reinterpret_cast<double*>(buf + off_pairs);
  p.partials   = reinterpret_cast<double*>(buf + off_part);
  cudaError_t e = ns > rg::kRankMax ? cudaMemsetAsync(p.regular, 1, sizeof(int), s) : cudaSuccess;
  if (e == cudaSuccess) {
    rg::ic_terms_kernel<<<term_blocks, rg::kPrepThreads, 0, s>>>(p);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess && tiles > 1) {
    rg::ic_tiles_kernel<<<4 * tiles, rg::kPrepThreads, 0, s>>>(p);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) {
    rg::ic_sums_kernel<<<4 * tiles, rg::kPrepThreads, 0, s>>>(p);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) {
    rg::ic_pair_kernel<<<dim3(col_blocks, splits), rg::kIcThreads, 0, s>>>(p);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = rg::launch_ic(K, p, dim3(grid, nslices), s);
  if (e == cudaSuccess) {
    rg::ic_reduce_kernel<<<col_blocks, dim3(32, 32), 0, s>>>(p, splits, grid, out);
    e = cudaGetLastError();
  }
  const cudaError_t ef = cudaFreeAsync(buf, s);
  if (e != cudaSuccess) {
    return rg::cuda_error(e, "rg_ic_spectrum launch");
  }
  RG_CUDA_TRY(ef);
  return RG_OK;
}

} // extern "C"

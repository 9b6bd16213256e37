// Particles<D>::energyDistribution (particles.cpp:189-260) on sm_103a.
//
// The reference computes Usqr = ux*ux + uy*uy + uz*uz in float, then the bin
// index through a double expression (double log10 of energy/emin, float log10
// of emax/emin), clamping out-of-range energies into bins 0 and n-1.  Because that
// index is a non-decreasing function of the float Usqr alone, the host finds,
// for every k, the smallest float Usqr whose index is >= k (binary search over
// float bit patterns with the reference's own expression).  The GPU computes
// Usqr with the same rounding steps, reads a lower bound of its bin from a table
// over cells of float bit patterns (the bin of each cell's smallest float) and
// steps over the thresholds inside the cell, so every particle lands in exactly
// the bin the reference picks and the counts are bit-exact.
//
// Log-spaced bins add float(1.0 / energy): for |u| energies that is the
// correctly rounded reciprocal of sqrtf(Usqr) (double rounding of one division
// of floats through double is innocuous); for sqrt(1 + Usqr) energies it is a
// double-float Newton step of rsqrt rounded to float.
//
// Only what the call asks for is accumulated: sums for log-spaced bins, counts otherwise or where
// they are asked for.  Sums of many particles over up to about 320 bins without counts
// (lane_warps): each of 16 lanes of a warp has its own copy of the bins in shared memory,
// [bin][copy], and the warp's halves add one after the other, so a particle is one conflict-free
// load, add and store.  Shared-memory atomics set the pace of the other kernel, which serves the
// rest: integer ones run at one lane per clock and SM on random bins, float ones as compare-and-swap
// loops.  FP32 sums are flushed to double-floats every kFlushLane particles of a lane (or
// kFlushParticles of a block), and blocks are summed in FP64 in a fixed order.
#include "pair_stage.cuh"
#include "rg_common.cuh"
#include "rg_internal.hpp"

#include <algorithm>
#include <cmath>
#include <cstring>
#include <limits>
#include <mutex>
#include <type_traits>
#include <vector>

namespace rg {

  namespace {

    constexpr int kHistThreads   = 256;
    // Copies of the FP32 sum bins, lane l adding into copy l mod kSumCopies: the float
    // shared-memory add retries while lanes of a warp hit the same bin, and energies
    // of a power law crowd a few bins (4 copies: 0.155 ms against 0.179 ms per call on
    // 3.3e7 particles; 16 copies were slower).
    constexpr int kSumCopies     = 4;
    constexpr int kHistMaxBins   = 4096;
    constexpr int kFlushParticles = 4096; // per block between flushes of the FP32 sums
    // Cells of the bin lookup: the finest cells of float bit patterns (bits >> shift)
    // such that [thr[1], the largest finite threshold] spans at most kMaxCells of them
    // (64 cells per octave for 200 log bins over five decades: at most one threshold
    // per cell).  Against an FP32 log2 estimate corrected both ways: 97.5 M against
    // 113.5 M warp instructions, 121.8 us against 130.8 us for 3.3e7 particles x 200 bins.
    constexpr int kMaxCells = 4096;

    // particles.cpp:224-253, the index of one particle given its float Usqr.
    std::size_t ref_energy_index(float Usqr, bool fourvel, float emin, float emax, std::size_t n) {
      const double energy = fourvel ? static_cast<double>(std::sqrt(Usqr)) : std::sqrt(1.0 + Usqr);
      if (energy < emin) {
        return 0;
      } else if (energy >= emax) {
        return n - 1;
      }
      const auto ei = static_cast<std::size_t>(static_cast<float>(n - 1) *
                                               std::fabs(std::log10(energy / emin)) /
                                               std::log10(emax / emin));
      return ei > n - 1 ? n - 1 : ei;
    }

    float bits_to_float(uint32_t b) {
      float f;
      std::memcpy(&f, &b, 4);
      return f;
    }

    // The lane kernel's cells are coarser (its table has 8 bytes a cell) and carry their first
    // threshold: each holds one at most, so a lookup is one load and one comparison.
    constexpr int kLaneCells   = 2048;
    constexpr int kLaneMaxWarps = 16;
    constexpr int kLaneCopies  = 16;   // copies of the bins per warp, lane l adding into copy l mod kLaneCopies
    constexpr int kLaneVectors = 4;    // groups of four particles in flight per thread
    constexpr int kFlushLane   = 512; // particles per lane between flushes
    constexpr uint32_t kLaneRow = sizeof(float) * kLaneCopies; // bytes of a bin's copies
    constexpr size_t kLaneSmem = 226 * 1024;

    struct HistParams {
      const float*    ux;
      const float*    uy;
      const float*    uz;
      int64_t         n;
      int             nbins;
      int             fourvel;
      int             log_spaced;
      const float*    thr;      // nbins thresholds: thr[k] = smallest Usqr with index >= k (thr[0] = 0)
      int             nan_index;
      const uint16_t* start;        // [ncells + 1]: 0, then the bin of each cell's smallest float
      int             cell_shift;   // cell of a float = its bit pattern >> cell_shift
      int             cell_base;    // cell of thr[1]
      int             ncells;
      const uint2*    lcells;       // lane kernel: [lncells + 2]: below thr[1], the cells, above the last threshold:
                                    // (kLaneRow x the bin of the cell's smallest float, next threshold's bits)
      int             lshift, lbase, lncells;
      unsigned long long* part_counts; // [grid][nbins], or null
      double*         part_sums;       // [grid][nbins], or null
    };

    // Bin of one particle: start[ci] is the bin of the smallest float of its cell (entry
    // 0 for cells below thr[1], the last entry for cells above the table), a lower bound
    // because the index is non-decreasing in Usqr; the thresholds between it and U are
    // stepped over (bounded).  Usqr >= 0, so its bit pattern orders like its value.
    __device__ __forceinline__ int bin_of(float U, const HistParams& p, const float* thr,
                                          const uint16_t* start) {
      if (U != U) {
        return p.nan_index;
      }
      int ci = static_cast<int>(__float_as_uint(U) >> p.cell_shift) - p.cell_base + 1;
      ci     = max(0, min(ci, p.ncells));
      int       g   = start[ci];
      const int nm1 = p.nbins - 1;
      for (int it = 0; it < p.nbins && g < nm1 && thr[g + 1] <= U; ++it) {
        ++g;
      }
      return g;
    }

    // float(1.0 / sqrt(1.0 + U)) without FP64: one Newton step in double-float.
    __device__ __forceinline__ float inv_sqrt_one_plus(float U) {
      if (!(U < 3.0e38f)) {
        return U == U ? 0.0f : U; // 1/sqrt(1 + inf) = 0; NaN stays NaN
      }
      const ff    s  = two_sum(1.0f, U);
      const float r0 = rsqrtf(s.hi);
      // e = 1 - s r0^2 in double-float, r = r0 + r0 e / 2
      const ff r2 = two_prod(r0, r0);
      const ff sr = ff_mul(s, r2);
      const float e = __fadd_rn(__fsub_rn(1.0f, sr.hi), -sr.lo);
      return __fmaf_rn(__fmul_rn(0.5f, r0), e, r0);
    }

    // 1/|u|: rsqrt and one Newton step (within an ulp; the reference rounds this value through
    // double, so the sums are compared with a tolerance anyway)
    __device__ __forceinline__ float inverse_energy(float U, int fourvel) {
      if (!fourvel) {
        return inv_sqrt_one_plus(U);
      }
      if (U > 0.0f && U < 3.0e38f) {
        const float r = rsqrtf(U);
        return __fmul_rn(r, __fmaf_rn(__fmul_rn(-0.5f * U, r), r, 1.5f));
      }
      return __frcp_rn(sqrtf(U)); // 0 -> inf, inf -> 0, NaN -> NaN
    }

    // t + (hi, lo) in double-float: infinite and NaN sums (an energy of 0) stay what they are, with no
    // low part.  The flushes below sum in this form because GB300 adds FP64 at 2 lanes a clock: with
    // FP64 sums 3.3e7 particles took 360 us over 2000 bins (now 198) and 161 over 600 (now 133).
    __device__ __forceinline__ ff sum_add(ff t, float hi, float lo) {
      const ff s = two_sum(t.hi, hi);
      return { s.hi, isfinite(s.hi) ? __fadd_rn(t.lo, __fadd_rn(s.lo, lo)) : 0.0f };
    }

    template <bool kSum, bool kCount>
    __global__ void __launch_bounds__(kHistThreads)
      histogram_kernel(const __grid_constant__ HistParams p) {
      extern __shared__ __align__(16) unsigned char smem[];
      const int nb      = p.nbins;
      float*    thr     = reinterpret_cast<float*>(smem);
      unsigned* cnt     = reinterpret_cast<unsigned*>(thr + nb);
      constexpr int kC = kSumCopies;
      float*    sum32   = reinterpret_cast<float*>(cnt + nb); // [kC][nb]
      float2*   total   = reinterpret_cast<float2*>(smem + (((2 + kC) * sizeof(float) * nb + 15) & ~size_t(15)));
      uint16_t* start   = reinterpret_cast<uint16_t*>(total + nb);
      for (int i = threadIdx.x; i < nb; i += blockDim.x) {
        thr[i]   = p.thr[i];
        cnt[i]   = 0u;
        total[i] = make_float2(0.0f, 0.0f);
      }
      for (int i = threadIdx.x; i < kC * nb; i += blockDim.x) {
        sum32[i] = 0.0f;
      }
      for (int i = threadIdx.x; i <= p.ncells; i += blockDim.x) {
        start[i] = p.start[i];
      }
      __syncthreads();
      float* sum_l = sum32 + (threadIdx.x & (kC - 1)) * nb;

      // contiguous range of particles per block, in rounds of kFlushParticles
      const int64_t G       = gridDim.x;
      const int64_t per     = ((p.n + G - 1) / G + 3) & ~int64_t(3);
      const int64_t begin   = min(p.n, per * blockIdx.x);
      const int64_t end     = min(p.n, begin + per);
      const bool    vec_ok  = ((reinterpret_cast<uintptr_t>(p.ux) | reinterpret_cast<uintptr_t>(p.uy) |
                            reinterpret_cast<uintptr_t>(p.uz)) & 15) == 0;

      for (int64_t r0 = begin; r0 < end; r0 += kFlushParticles) {
        const int64_t r1 = min(end, r0 + kFlushParticles);
        auto          one = [&](float x, float y, float z) {
          const float U = __fadd_rn(__fadd_rn(__fmul_rn(x, x), __fmul_rn(y, y)), __fmul_rn(z, z));
          const int   k = bin_of(U, p, thr, start);
          if (kCount) {
            atomicAdd(&cnt[k], 1u);
          }
          if (kSum) {
            const float v = inverse_energy(U, p.fourvel);
            atomicAdd(&sum_l[k], v);
          }
        };
        if (vec_ok) {
          // 4 particles per thread with 128-bit loads (begin and per are multiples of 4)
          const int64_t nv = (r1 - r0) / 4;
          for (int64_t v = threadIdx.x; v < nv; v += blockDim.x) {
            const int64_t i  = r0 + 4 * v;
            const float4  X  = __ldcs(reinterpret_cast<const float4*>(p.ux + i));
            const float4  Y  = __ldcs(reinterpret_cast<const float4*>(p.uy + i));
            const float4  Z  = __ldcs(reinterpret_cast<const float4*>(p.uz + i));
            one(X.x, Y.x, Z.x);
            one(X.y, Y.y, Z.y);
            one(X.z, Y.z, Z.z);
            one(X.w, Y.w, Z.w);
          }
          for (int64_t i = r0 + 4 * nv + threadIdx.x; i < r1; i += blockDim.x) {
            one(p.ux[i], p.uy[i], p.uz[i]);
          }
        } else {
          for (int64_t i = r0 + threadIdx.x; i < r1; i += blockDim.x) {
            one(p.ux[i], p.uy[i], p.uz[i]);
          }
        }
        if (kSum) {
          __syncthreads();
          for (int i = threadIdx.x; i < nb; i += blockDim.x) {
            ff t { total[i].x, total[i].y };
#pragma unroll
            for (int c = 0; c < kC; ++c) {
              t                 = sum_add(t, sum32[c * nb + i], 0.0f);
              sum32[c * nb + i] = 0.0f;
            }
            total[i] = make_float2(t.hi, t.lo);
          }
        }
        __syncthreads();
      }
      for (int i = threadIdx.x; i < nb; i += blockDim.x) {
        if (kCount) {
          p.part_counts[static_cast<int64_t>(blockIdx.x) * nb + i] = cnt[i];
        }
        if (kSum) {
          p.part_sums[static_cast<int64_t>(blockIdx.x) * nb + i] = static_cast<double>(total[i].x) + static_cast<double>(total[i].y);
        }
      }
    }

    // Energies whose reciprocal the packed expressions below give: 2^-126 <= Usqr < 2^100, as an
    // interval of bit patterns (which leaves out NaN too).
    constexpr uint32_t kOrdinaryMin  = 0x00800000u;
    constexpr uint32_t kOrdinarySpan = 0x71800000u - kOrdinaryMin;

    __device__ __forceinline__ f2 rsqrt2(float a, float b) {
      asm("rsqrt.approx.ftz.f32 %0, %0;" : "+f"(a));
      asm("rsqrt.approx.ftz.f32 %0, %0;" : "+f"(b));
      return pack2(a, b);
    }

    // inv_sqrt_one_plus of two: r + r (1 - s r^2) / 2 with s = 1 + U in double-float.  r^2 = h + l and
    // s.hi h - 1 are exact or rounded once, so the correction keeps its leading digits.
    __device__ __forceinline__ f2 inv_sqrt_one_plus2(f2 U) {
      const ff2 s = two_sum2(set2(1.0f), U);
      float     a, b;
      unpack2(s.hi, a, b);
      const f2 r = rsqrt2(a, b);
      const f2 h = mul2(r, r), l = fma2(r, r, neg2(h));
      const f2 e = add2(fma2(s.hi, h, set2(-1.0f)), fma2(s.hi, l, mul2(s.lo, h))); // s r^2 - 1
      return fma2(mul2(r, set2(-0.5f)), e, r);
    }

    // shared [k0] += v0, then [k1] += v1 (which may be the same bin) where `on`
    __device__ __forceinline__ void add_pair(uint32_t k0, uint32_t k1, float v0, float v1, bool on) {
      asm volatile("{\n"
                   "  .reg .pred p, q;\n"
                   "  .reg .f32 a, b;\n"
                   "  setp.ne.u32 p, %4, 0;\n"
                   "  setp.eq.u32 q, %0, %1;\n"
                   "  @p ld.shared.f32 a, [%0];\n"
                   "  @p ld.shared.f32 b, [%1];\n"
                   "  add.rn.f32 a, a, %2;\n"
                   "  selp.f32 b, a, b, q;\n"
                   "  add.rn.f32 b, b, %3;\n"
                   "  @p st.shared.f32 [%0], a;\n"
                   "  @p st.shared.f32 [%1], b;\n"
                   "}" ::"r"(k0), "r"(k1), "f"(v0), "f"(v1), "r"(static_cast<uint32_t>(on))
                   : "memory");
    }

    // Any particle's bin by stepping over the thresholds from g (energies of 0, infinity and NaN).
    __device__ __noinline__ int bin_by_steps(float U, const HistParams& p, const float* thr, int g) {
      if (U != U) {
        return p.nan_index;
      }
      while (g < p.nbins - 1 && thr[g + 1] <= U) {
        ++g;
      }
      return g;
    }

    // Shared memory of the lane kernel with `warps` warps.
    size_t lane_smem(int nb, int ncells, int warps) {
      return (sizeof(float2) + sizeof(float)) * nb + sizeof(uint2) * (ncells + 2) +
             sizeof(float) * kLaneCopies * static_cast<size_t>(nb) * warps + 16;
    }

    // Shared memory of the atomics kernel.
    size_t atomics_smem(int nb, int ncells) {
      return (((2 + kSumCopies) * sizeof(float) * nb + 15) & ~size_t(15)) + sizeof(float2) * nb + sizeof(uint16_t) * (ncells + 1);
    }

    // Warps of the lane kernel, or 0 where the atomics are faster: with fewer than ten warps on an SM
    // latencies are not hidden, and clearing and summing the copies takes as long as a million
    // particles.  Per call, sums of |u|^-1 over log bins, lanes against atomics: 3.3e7 particles x 25
    // bins 97 / 185 us, 50: 92 / 155, 100: 94 / 139, 200: 89 / 128, 300 (10 warps): 114 / 128, 380
    // (8 warps): 138 / 128; 200 bins x 8e6: 37.9 / 51.1, 3e6: 27.6 / 30.9, 1e6: 23.4 / 23.2.  Counts stay
    // with the integer atomics (200 bins: 77); streams off a 16-byte boundary,
    // and bins so uneven that a cell holds several thresholds, go to the atomics kernel too.
    constexpr int     kLaneMinWarps     = 10;
    constexpr int64_t kLaneMinParticles = 2000000;

    int lane_warps(const float* ux, const float* uy, const float* uz, int64_t n, int nb, int ncells) {
      const size_t tables = lane_smem(nb, ncells, 0);
      const bool   aligned = ((reinterpret_cast<uintptr_t>(ux) | reinterpret_cast<uintptr_t>(uy) |
                             reinterpret_cast<uintptr_t>(uz)) & 15) == 0;
      if (!aligned || n < kLaneMinParticles || tables >= kLaneSmem) {
        return 0;
      }
      const size_t w = (kLaneSmem - tables) / (sizeof(float) * kLaneCopies * nb);
      return w < static_cast<size_t>(kLaneMinWarps) ? 0 : static_cast<int>(std::min<size_t>(w, kLaneMaxWarps));
    }

    // What bounds it: latency.  200 bins leave room for 16 warps on an SM (copies: 12.8 KB each).  3.3e7
    // particles x 200 bins with 1/|u|: 89 us a call (4.4 TB/s) against 128 us with atomics and 139 us with
    // atomics and FP64 flushes.  A copy per lane leaves 8 warps: 121 us; two groups of four at a
    // time spill: 123 us before the flushes were in double-floats, one group 103 us.
    __global__ void __launch_bounds__(32 * kLaneMaxWarps) histogram_lane_kernel(const __grid_constant__ HistParams p) {
      extern __shared__ __align__(16) unsigned char smem[];
      const int nb = p.nbins, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
      float2*   total = reinterpret_cast<float2*>(smem);
      uint2*    cells = reinterpret_cast<uint2*>(total + nb);
      float*    thr   = reinterpret_cast<float*>(cells + p.lncells + 2);
      float*    copies = reinterpret_cast<float*>((reinterpret_cast<uintptr_t>(thr + nb) + 15) & ~uintptr_t(15));
      const int per    = kLaneCopies * nb;
      float*    mine   = copies + warp * per; // [nb][kLaneCopies]
      for (int i = threadIdx.x; i < nb; i += blockDim.x) {
        thr[i]   = p.thr[i];
        total[i] = make_float2(0.0f, 0.0f);
      }
      for (int i = threadIdx.x; i < p.lncells + 2; i += blockDim.x) {
        cells[i] = p.lcells[i];
      }
      for (int i = threadIdx.x; i < warps * per / 4; i += blockDim.x) {
        reinterpret_cast<uint4*>(copies)[i] = make_uint4(0u, 0u, 0u, 0u);
      }
      __syncthreads();

      // 2 N particles of a lane: the bins and values of all of them first, then the additions in
      // pairs (the two of a pair may share a bin).
      const uint32_t copy0 = static_cast<uint32_t>(__cvta_generic_to_shared(mine + (lane & (kLaneCopies - 1))));
      const uint32_t upper = lane >> 4; // lanes l and l + 16 share a copy: the lower ones add first
      const uint32_t cell0 = static_cast<uint32_t>(__cvta_generic_to_shared(cells)) - 8u * static_cast<uint32_t>(p.lbase - 1);
      const int      cmin = p.lbase - 1, cmax = p.lbase + p.lncells;
      const bool     fourvel = p.fourvel != 0;
      auto           add     = [&](auto const& x, auto const& y, auto const& z, auto count_tag) {
        constexpr int N = decltype(count_tag)::value;
        float         u[2 * N], v[2 * N];
        uint32_t      k[2 * N];
        uint32_t      far = 0u;
#pragma unroll
        for (int j = 0; j < N; ++j) {
          // single products: the compiler contracts a packed product and sum, whatever their rounding
          // modifiers, and Usqr has to be the reference's
          float x0, x1, y0, y1, z0, z1;
          unpack2(x[j], x0, x1);
          unpack2(y[j], y0, y1);
          unpack2(z[j], z0, z1);
          u[2 * j]     = __fadd_rn(__fadd_rn(__fmul_rn(x0, x0), __fmul_rn(y0, y0)), __fmul_rn(z0, z0));
          u[2 * j + 1] = __fadd_rn(__fadd_rn(__fmul_rn(x1, x1), __fmul_rn(y1, y1)), __fmul_rn(z1, z1));
          const f2 U   = pack2(u[2 * j], u[2 * j + 1]);
#pragma unroll
          for (int h = 2 * j; h < 2 * j + 2; ++h) {
            const uint32_t bits = __float_as_uint(u[h]);
            uint32_t       cx, cy;
            asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(cx), "=r"(cy) : "r"(cell0 + 8u * static_cast<uint32_t>(max(cmin, min(static_cast<int>(bits >> p.lshift), cmax)))));
            k[h] = copy0 + cx + (u[h] >= __uint_as_float(cy) ? kLaneRow : 0u);
            far = max(far, bits - kOrdinaryMin);
          }
          if (fourvel) { // inverse_energy of an ordinary U
            const f2 r = rsqrt2(u[2 * j], u[2 * j + 1]);
            unpack2(mul2(r, fma2(mul2(mul2(U, set2(-0.5f)), r), r, set2(1.5f))), v[2 * j], v[2 * j + 1]);
          } else {
            unpack2(inv_sqrt_one_plus2(U), v[2 * j], v[2 * j + 1]);
          }
        }
        if (far >= kOrdinarySpan) {
#pragma unroll
          for (int h = 0; h < 2 * N; ++h) {
            const uint32_t bits = __float_as_uint(u[h]);
            const int      ci   = max(cmin, min(static_cast<int>(bits >> p.lshift), cmax)) - cmin;
            k[h] = copy0 + kLaneRow * static_cast<uint32_t>(bin_by_steps(u[h], p, thr, static_cast<int>(cells[ci].x / kLaneRow)));
            v[h] = inverse_energy(u[h], p.fourvel);
          }
        }
#pragma unroll
        for (uint32_t half = 0; half < 2; ++half) {
#pragma unroll
          for (int j = 0; j < N; ++j) {
            add_pair(k[2 * j], k[2 * j + 1], v[2 * j], v[2 * j + 1], upper == half);
          }
          __syncwarp();
        }
      };
      auto add_one = [&](bool live, float x, float y, float z) {
        uint32_t at = copy0;
        float    v  = 0.0f;
        if (live) {
          const float U  = __fadd_rn(__fadd_rn(__fmul_rn(x, x), __fmul_rn(y, y)), __fmul_rn(z, z));
          const int   ci = max(cmin, min(static_cast<int>(__float_as_uint(U) >> p.lshift), cmax)) - cmin;
          at = copy0 + kLaneRow * static_cast<uint32_t>(bin_by_steps(U, p, thr, static_cast<int>(cells[ci].x / kLaneRow)));
          v  = inverse_energy(U, p.fourvel);
        }
        __syncwarp();
#pragma unroll
        for (uint32_t half = 0; half < 2; ++half) {
          if (live && upper == half) {
            float a;
            asm volatile("ld.shared.f32 %0, [%1];" : "=f"(a) : "r"(at) : "memory");
            asm volatile("st.shared.f32 [%0], %1;" ::"r"(at), "f"(__fadd_rn(a, v)) : "memory");
          }
          __syncwarp();
        }
      };
      // The lanes' copies into the block's totals: a thread sums the copies of its bins in four
      // chains (starting at a different lane per bin, so that a warp's reads hit different banks),
      // then the warps'.
      auto flush = [&]() {
        __syncwarp();
        for (int b = lane; b < nb; b += 32) {
          ff t[4];
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            t[c] = ff { 0.0f, 0.0f };
          }
#pragma unroll 2
          for (int l = 0; l < kLaneCopies; l += 4) {
#pragma unroll
            for (int c = 0; c < 4; ++c) {
              const int at = b * kLaneCopies + ((l + c + b) & (kLaneCopies - 1));
              t[c]         = sum_add(t[c], mine[at], 0.0f);
              mine[at]     = 0.0f;
            }
          }
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            mine[b * kLaneCopies + 2 * c]     = t[c].hi;
            mine[b * kLaneCopies + 2 * c + 1] = t[c].lo;
          }
        }
        __syncthreads();
        // four threads a bin sum the warps' pairs of one chain each
        for (int i = threadIdx.x; i < ((4 * nb + 31) & ~31); i += blockDim.x) {
          const int b = i >> 2, c = i & 3;
          ff        t { 0.0f, 0.0f };
          if (b < nb) {
            for (int w = 0; w < warps; ++w) {
              float* m = copies + w * per + b * kLaneCopies + 2 * c;
              t        = sum_add(t, m[0], m[1]);
              m[0]     = 0.0f;
              m[1]     = 0.0f;
            }
          }
#pragma unroll
          for (int o = 1; o < 4; o <<= 1) {
            t = sum_add(t, __shfl_xor_sync(0xffffffffu, t.hi, o), __shfl_xor_sync(0xffffffffu, t.lo, o));
          }
          if (b < nb && c == 0) {
            t        = sum_add(t, total[b].x, total[b].y);
            total[b] = make_float2(t.hi, t.lo);
          }
        }
        __syncthreads();
      };

      const int64_t T = static_cast<int64_t>(gridDim.x) * blockDim.x;
      const int64_t t = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
      const int64_t nv = p.n / 4; // groups of four, loaded as 16 bytes (lane_warps asks for the alignment)
      int           since = 0;    // particles of a lane since the last flush (the same in every thread)
      // kLaneVectors groups in flight: a group's registers are loaded again as soon as it is added
      float4 X[kLaneVectors], Y[kLaneVectors], Z[kLaneVectors];
      auto   load = [&](int k, int64_t v) {
        if (v < nv) {
          X[k] = __ldcs(reinterpret_cast<const float4*>(p.ux) + v);
          Y[k] = __ldcs(reinterpret_cast<const float4*>(p.uy) + v);
          Z[k] = __ldcs(reinterpret_cast<const float4*>(p.uz) + v);
        }
      };
#pragma unroll
      for (int k = 0; k < kLaneVectors; ++k) {
        load(k, k * T + t);
      }
      for (int64_t v0 = 0; v0 < nv; v0 += kLaneVectors * T) { // uniform over the grid
#pragma unroll
        for (int k = 0; k < kLaneVectors; ++k) {
          const int64_t v    = v0 + k * T + t;
          const f2      x[2] = { pack2(X[k].x, X[k].y), pack2(X[k].z, X[k].w) };
          const f2      y[2] = { pack2(Y[k].x, Y[k].y), pack2(Y[k].z, Y[k].w) };
          const f2      z[2] = { pack2(Z[k].x, Z[k].y), pack2(Z[k].z, Z[k].w) };
          if (v - lane + 31 < nv) { // the whole warp has a group
            add(x, y, z, std::integral_constant<int, 2> {});
          } else {
#pragma unroll 1
            for (int i = 0; i < 4; ++i) {
              const int64_t g = 4 * v + i;
              add_one(v < nv, v < nv ? p.ux[g] : 0.0f, v < nv ? p.uy[g] : 0.0f, v < nv ? p.uz[g] : 0.0f);
            }
          }
          load(k, v + kLaneVectors * T);
        }
        since += 4 * kLaneVectors;
        if (since >= kFlushLane) {
          flush();
          since = 0;
        }
      }
      { // the remainder
        const int64_t i    = 4 * nv + t;
        const bool    live = i < p.n;
        add_one(live, live ? p.ux[i] : 0.0f, live ? p.uy[i] : 0.0f, live ? p.uz[i] : 0.0f);
      }
      flush();
      for (int b = threadIdx.x; b < nb; b += blockDim.x) {
        p.part_sums[static_cast<int64_t>(blockIdx.x) * nb + b] = static_cast<double>(total[b].x) + static_cast<double>(total[b].y);
      }
    }

    // Block (32 bins x 32 row groups): row group y sums block partials y, y + 32, ...
    // then the groups are combined in order (deterministic).
    constexpr int kHistReduceRows = 32;

    __global__ void __launch_bounds__(32 * kHistReduceRows)
      histogram_reduce_kernel(const unsigned long long* __restrict__ pc, const double* __restrict__ ps,
                              int grid, int nbins, int log_spaced, float* __restrict__ hist,
                              unsigned long long* __restrict__ counts) {
      __shared__ unsigned long long c_part[kHistReduceRows][33];
      __shared__ double             s_part[kHistReduceRows][33];
      const int k  = blockIdx.x * 32 + threadIdx.x;
      const int ty = threadIdx.y;
      unsigned long long c = 0;
      double             s = 0.0;
      if (k < nbins) {
        // unrolled so that several rows' loads are in flight (the adds stay in row order)
#pragma unroll 8
        for (int b = ty; b < grid; b += kHistReduceRows) {
          c += pc ? pc[static_cast<int64_t>(b) * nbins + k] : 0ull;
          s += ps ? ps[static_cast<int64_t>(b) * nbins + k] : 0.0;
        }
      }
      c_part[ty][threadIdx.x] = c;
      s_part[ty][threadIdx.x] = s;
      __syncthreads();
      if (ty != 0 || k >= nbins) {
        return;
      }
      for (int y = 1; y < kHistReduceRows; ++y) {
        c += c_part[y][threadIdx.x];
        s += s_part[y][threadIdx.x];
      }
      hist[k] = log_spaced ? __double2float_rn(s) : static_cast<float>(c);
      if (counts) {
        counts[k] = c;
      }
    }

  } // namespace

  // Thresholds thr[k] (k = 1..n-1): the smallest non-negative float Usqr whose
  // reference index is >= k (+inf if none); thr[0] = 0.  Exposed for tests.
  void energy_thresholds(const float* bins, int n, bool fourvel, std::vector<float>& thr,
                         int& nan_index, float& emin, float& emax) {
    emin = std::numeric_limits<float>::max();
    emax = std::numeric_limits<float>::lowest();
    for (int i = 0; i < n; ++i) {
      emin = std::min(emin, bins[i]);
      emax = std::max(emax, bins[i]);
    }
    thr.assign(n, 0.0f);
    const uint32_t inf_bits = 0x7f800000u;
    for (int k = 1; k < n; ++k) {
      // smallest bit pattern b in [0, inf] with index(b) >= k
      uint32_t lo = 0, hi = inf_bits;
      if (ref_energy_index(bits_to_float(hi), fourvel, emin, emax, n) < static_cast<std::size_t>(k)) {
        thr[k] = std::numeric_limits<float>::infinity();
        continue;
      }
      while (lo < hi) {
        const uint32_t mid = lo + (hi - lo) / 2;
        if (ref_energy_index(bits_to_float(mid), fourvel, emin, emax, n) >= static_cast<std::size_t>(k)) {
          hi = mid;
        } else {
          lo = mid + 1;
        }
      }
      thr[k] = bits_to_float(lo);
    }
    nan_index = static_cast<int>(
      ref_energy_index(std::numeric_limits<float>::quiet_NaN(), fourvel, emin, emax, n));
  }

  namespace {

    // Thresholds of recently used bin sets (the host binary search costs far more
    // than the histogram kernel for small particle counts), with one device copy per
    // GPU that used them, so a call copies nothing to the device and need not wait
    // for a host buffer; keyed on the bin values and the energy definition, at most
    // kThrCacheEntries kept.
    struct ThrEntry {
      std::vector<float>                  bins, thr;
      bool                                fourvel   = true;
      int                                 nan_index = 0;
      float                               emin = 0, emax = 0;
      std::vector<uint16_t>               start; // cell table (see bin_of)
      int                                 cell_shift = 0, cell_base = 0, ncells = 0;
      std::vector<uint2>                  lcells; // cell table of the lane kernel
      int                                 lshift = 0, lbase = 0, lncells = 0;
      std::vector<std::pair<int, float*>> dev; // (device, the lane kernel's cells, thresholds, cell table there)
    };

    uint32_t float_bits(float f) {
      uint32_t b;
      std::memcpy(&b, &f, 4);
      return b;
    }

    // The cell table over [thr[1], the largest finite threshold]: the smallest shift
    // that keeps at most kMaxCells cells; start[0] = 0 (cells below thr[1]) and
    // start[i] = the number of thresholds thr[1..n-1] <= the smallest float of cell
    // cell_base + i - 1, i.e. that float's bin.  No finite thr[1]: no cells, every
    // particle starts from bin 0.
    void make_cells(ThrEntry& e) {
      const int n = static_cast<int>(e.thr.size());
      e.start.assign(1, 0);
      e.cell_shift = 0;
      e.cell_base  = 0;
      e.ncells     = 0;
      if (n < 2 || !std::isfinite(e.thr[1])) {
        return;
      }
      const uint32_t lo = float_bits(e.thr[1]);
      uint32_t       hi = lo;
      for (int k = 1; k < n; ++k) {
        if (std::isfinite(e.thr[k])) {
          hi = float_bits(e.thr[k]);
        }
      }
      int sh = 0;
      while (sh < 31 && (hi >> sh) - (lo >> sh) + 1 > static_cast<uint32_t>(kMaxCells)) {
        ++sh;
      }
      e.cell_shift = sh;
      e.cell_base  = static_cast<int>(lo >> sh);
      e.ncells     = static_cast<int>((hi >> sh) - (lo >> sh) + 1);
      e.start.resize(static_cast<std::size_t>(e.ncells) + 1);
      int k = 1; // thr[1..k-1] <= the current cell's smallest float
      for (int i = 1; i <= e.ncells; ++i) {
        const float low = bits_to_float(static_cast<uint32_t>(e.cell_base + i - 1) << sh);
        while (k < n && e.thr[k] <= low) {
          ++k;
        }
        e.start[i] = static_cast<uint16_t>(k - 1);
      }
    }

    // The lane kernel's cells from the first threshold above 0 to the last finite one (see
    // HistParams::lcells); none, and no lane kernel, where a cell would hold several thresholds.
    void make_lane_cells(ThrEntry& e) {
      const int      n   = static_cast<int>(e.thr.size());
      const uint32_t inf = 0x7f800000u;
      int            zero = 0, fin = 0; // thresholds thr[1..zero] are 0, thr[1..fin] finite
      while (fin + 1 < n && std::isfinite(e.thr[fin + 1])) {
        ++fin;
      }
      while (zero < fin && e.thr[zero + 1] == 0.0f) {
        ++zero;
      }
      e.lshift  = 0;
      e.lbase   = 0;
      e.lncells = 0;
      e.lcells.assign(2, make_uint2(kLaneRow * static_cast<uint32_t>(zero), inf));
      if (fin == zero) { // no threshold above 0: one bin for every finite energy
        return;
      }
      const uint32_t lo = float_bits(e.thr[zero + 1]), hi = float_bits(e.thr[fin]);
      while ((hi >> e.lshift) - (lo >> e.lshift) + 1 > static_cast<uint32_t>(kLaneCells)) {
        ++e.lshift;
      }
      e.lbase   = static_cast<int>(lo >> e.lshift);
      e.lncells = static_cast<int>((hi >> e.lshift) - (lo >> e.lshift) + 1);
      e.lcells.resize(static_cast<std::size_t>(e.lncells) + 2);
      int k = 1; // thr[1..k-1] <= the current cell's smallest float
      for (int i = 1; i <= e.lncells; ++i) {
        const uint32_t first = static_cast<uint32_t>(e.lbase + i - 1) << e.lshift;
        while (k <= fin && float_bits(e.thr[k]) <= first) {
          ++k;
        }
        const uint64_t next = static_cast<uint64_t>(first) + (uint64_t(1) << e.lshift);
        if (k + 1 <= fin && float_bits(e.thr[k + 1]) < next) {
          e.lcells.clear();
          return;
        }
        e.lcells[i] = make_uint2(kLaneRow * static_cast<uint32_t>(k - 1), k <= fin ? float_bits(e.thr[k]) : inf);
      }
      e.lcells[e.lncells + 1] = make_uint2(kLaneRow * static_cast<uint32_t>(fin), inf);
    }

    constexpr std::size_t kThrCacheEntries = 16;

    std::mutex& thr_mutex() {
      static std::mutex m;
      return m;
    }

    std::vector<ThrEntry>& thr_cache() { // most recent last
      static std::vector<ThrEntry> c;
      return c;
    }

    // Frees the device copies of an entry; a kernel of any stream may still read them,
    // so each device is synchronised first (entries are evicted rarely).
    void free_entry(ThrEntry& e) {
      int cur = 0;
      cudaGetDevice(&cur);
      for (auto& d : e.dev) {
        cudaSetDevice(d.first);
        cudaDeviceSynchronize();
        cudaFree(d.second);
      }
      cudaSetDevice(cur);
      e.dev.clear();
    }

  } // namespace

  // What the histogram kernel needs of a bin set, on the current device.
  struct DeviceBins {
    const float*    thr   = nullptr;
    const uint16_t* start = nullptr;
    const uint2*    lcells = nullptr;
    int             lshift = 0, lbase = 0, lncells = 0;
    int             nan_index = 0, cell_shift = 0, cell_base = 0, ncells = 0;
  };

  // Thresholds and cell table of a bin set on the current device.  The caller holds thr_mutex until the
  // kernel that reads them is queued: another thread's bin set may evict this one, which waits for the
  // device and frees it.
  int device_thresholds(const float* bins, int n, bool fourvel, DeviceBins& out) {
    int device = 0;
    RG_CUDA_TRY(cudaGetDevice(&device));
    auto&                       cache = thr_cache();
    auto                        it    = cache.begin();
    for (; it != cache.end(); ++it) {
      if (it->fourvel == fourvel && static_cast<int>(it->bins.size()) == n &&
          std::memcmp(it->bins.data(), bins, sizeof(float) * n) == 0) {
        break;
      }
    }
    if (it == cache.end()) {
      ThrEntry e;
      energy_thresholds(bins, n, fourvel, e.thr, e.nan_index, e.emin, e.emax);
      make_cells(e);
      make_lane_cells(e);
      e.bins.assign(bins, bins + n);
      e.fourvel = fourvel;
      if (cache.size() >= kThrCacheEntries) {
        free_entry(cache.front());
        cache.erase(cache.begin());
      }
      cache.push_back(std::move(e));
      it = cache.end() - 1;
    } else {
      std::rotate(it, it + 1, cache.end());
      it = cache.end() - 1;
    }
    ThrEntry& e = *it;
    float*    p = nullptr;
    for (auto& d : e.dev) {
      if (d.first == device) {
        p = d.second;
      }
    }
    if (!p) {
      const size_t lbytes = sizeof(uint2) * e.lcells.size();
      RG_CUDA_TRY(cudaMalloc(&p, lbytes + sizeof(float) * n + sizeof(uint16_t) * e.start.size()));
      float*      t   = reinterpret_cast<float*>(reinterpret_cast<unsigned char*>(p) + lbytes);
      cudaError_t err = cudaMemcpy(p, e.lcells.data(), lbytes, cudaMemcpyHostToDevice);
      if (err == cudaSuccess) {
        err = cudaMemcpy(t, e.thr.data(), sizeof(float) * n, cudaMemcpyHostToDevice);
      }
      if (err == cudaSuccess) {
        err = cudaMemcpy(t + n, e.start.data(), sizeof(uint16_t) * e.start.size(), cudaMemcpyHostToDevice);
      }
      if (err != cudaSuccess) {
        cudaFree(p);
        return cuda_error(err, "threshold copy");
      }
      e.dev.emplace_back(device, p);
    }
    out.lcells     = e.lcells.empty() ? nullptr : reinterpret_cast<const uint2*>(p);
    out.thr        = reinterpret_cast<const float*>(reinterpret_cast<const uint2*>(p) + e.lcells.size());
    out.start      = reinterpret_cast<const uint16_t*>(out.thr + n);
    out.lshift     = e.lshift;
    out.lbase      = e.lbase;
    out.lncells    = e.lncells;
    out.nan_index  = e.nan_index;
    out.cell_shift = e.cell_shift;
    out.cell_base  = e.cell_base;
    out.ncells     = e.ncells;
    return RG_OK;
  }

  void free_threshold_cache() {
    std::lock_guard<std::mutex> lock(thr_mutex());
    for (auto& e : thr_cache()) {
      free_entry(e);
    }
    thr_cache().clear();
  }

} // namespace rg

extern "C" {

int rg_energy_thresholds(const float* bins, int32_t nbins, int32_t fourvel, float* thr,
                         int32_t* nan_index) {
  if (nbins < 1 || !bins || !thr) {
    return rg::set_error(RG_ERR_ARGUMENT, "rg_energy_thresholds: bad arguments");
  }
  std::vector<float> t;
  int                ni = 0;
  float              emin, emax;
  rg::energy_thresholds(bins, nbins, fourvel != 0, t, ni, emin, emax);
  std::copy(t.begin(), t.end(), thr);
  if (nan_index) {
    *nan_index = ni;
  }
  return RG_OK;
}

int rg_energy_distribution(const float* ux, const float* uy, const float* uz, int64_t n,
                           const float* bins, int32_t nbins, int32_t log_spaced, int32_t fourvel,
                           float* hist, uint64_t* counts, void* stream) {
  rg::NvtxRange nvtx_range("ComputeEnergyDistribution");
  rg::clear_error();
  if (nbins < 1 || !bins || !hist || n < 0 || (n > 0 && (!ux || !uy || !uz))) {
    return rg::set_error(RG_ERR_ARGUMENT, "rg_energy_distribution: bad arguments");
  }
  if (nbins > rg::kHistMaxBins) {
    return rg::set_error(RG_ERR_UNSUPPORTED, "energyDistribution supports at most 4096 bins");
  }
  auto           s = static_cast<cudaStream_t>(stream);
  std::lock_guard<std::mutex> lock(rg::thr_mutex()); // see device_thresholds
  rg::DeviceBins              db;
  RG_TRY(rg::device_thresholds(bins, nbins, fourvel != 0, db));

  rg::DeviceContext* ctx = nullptr;
  RG_TRY(rg::context(&ctx));
  // what is accumulated, and by which kernel
  const bool need_sum = log_spaced != 0, need_count = !need_sum || counts != nullptr;
  const int  warps    = need_count || !db.lcells ? 0 : rg::lane_warps(ux, uy, uz, n, nbins, db.lncells);
  size_t     smem     = 0;
  int        G        = 0;
  auto       kernel   = !need_sum    ? rg::histogram_kernel<false, true>
                        : need_count ? rg::histogram_kernel<true, true>
                                     : rg::histogram_kernel<true, false>;
  if (warps > 0) {
    static std::atomic<uint64_t> configured { 0 };
    RG_CUDA_TRY(rg::ensure_max_dynamic_smem(rg::histogram_lane_kernel, static_cast<int>(rg::kLaneSmem), configured));
    smem = rg::lane_smem(nbins, db.lncells, warps);
    G    = ctx->sms * std::max(1, std::min(static_cast<int>(rg::kLaneSmem / smem), 2048 / (32 * rg::kLaneMaxWarps)));
  } else {
    smem = rg::atomics_smem(nbins, db.ncells);
    // the limit once for all sizes: set to a call's own size it may be lowered by another thread's call
    // before the launch
    static std::atomic<uint64_t> configured[3];
    RG_CUDA_TRY(rg::ensure_max_dynamic_smem(kernel, static_cast<int>(rg::atomics_smem(rg::kHistMaxBins, rg::kMaxCells)),
                                            configured[!need_sum ? 0 : need_count ? 1 : 2]));
    int per_sm = 0;
    RG_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, rg::kHistThreads, smem));
    per_sm = std::max(1, std::min(per_sm, 8));
    // at least 4096 particles a block, or 1024 while that leaves room on the chip (a call on 1e3
    // particles 20 -> 14 us, 1e4 24 -> 13, 1e5 24 -> 15, 1e6 28 -> 23)
    const int64_t want = std::max<int64_t>({ 1, (n + 4095) / 4096, std::min<int64_t>((n + 1023) / 1024, 2 * ctx->sms) });
    G = static_cast<int>(std::min<int64_t>(want, static_cast<int64_t>(ctx->sms) * per_sm));
  }

  // one stream-ordered allocation for the per-block partials
  const size_t   rows   = static_cast<size_t>(G) * nbins;
  const size_t   off_ps = need_count ? sizeof(unsigned long long) * rows : 0;
  const size_t   bytes  = off_ps + (need_sum ? sizeof(double) * rows : 0);
  unsigned char* buf    = nullptr;
  RG_TRY(rg::scratch_alloc(reinterpret_cast<void**>(&buf), bytes, s));

  rg::HistParams p {};
  p.ux         = ux;
  p.uy         = uy;
  p.uz         = uz;
  p.n          = n;
  p.nbins      = nbins;
  p.fourvel    = fourvel ? 1 : 0;
  p.log_spaced = log_spaced ? 1 : 0;
  p.thr        = db.thr;
  p.nan_index  = db.nan_index;
  p.start      = db.start;
  p.cell_shift = db.cell_shift;
  p.cell_base  = db.cell_base;
  p.ncells     = db.ncells;
  p.lcells     = db.lcells;
  p.lshift     = db.lshift;
  p.lbase      = db.lbase;
  p.lncells    = db.lncells;
  p.part_counts = need_count ? reinterpret_cast<unsigned long long*>(buf) : nullptr;
  p.part_sums   = need_sum ? reinterpret_cast<double*>(buf + off_ps) : nullptr;
  if (warps > 0) {
    rg::histogram_lane_kernel<<<G, 32 * warps, smem, s>>>(p);
  } else {
    kernel<<<G, rg::kHistThreads, smem, s>>>(p);
  }
  RG_CUDA_TRY(cudaGetLastError());
  rg::histogram_reduce_kernel<<<(nbins + 31) / 32, dim3(32, rg::kHistReduceRows), 0, s>>>(
    p.part_counts, p.part_sums, G, nbins, p.log_spaced, hist,
    reinterpret_cast<unsigned long long*>(counts));
  RG_CUDA_TRY(cudaGetLastError());
  RG_CUDA_TRY(cudaFreeAsync(buf, s));
  return RG_OK;
}

} // extern "C"

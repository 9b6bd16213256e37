// Particle synchrotron spectrum by interval moments (reference table).
//
// Reference path: SynchrotronSpectrum<D> (synchrotron.cpp:107-145) summing
// sync::Kernel<D>::operator() (synchrotron.hpp:145-172) over every (particle,
// photon bin) pair, with F from the 200-point table interpolated linearly in
// log x (InterpolateTabulatedFunction<true>, tabulation.hpp:19-53).
//
// The spectrum is the same sum, S_b = e_b sum_p A_p f(P_b - Q_p), of the same
// function f of the same fixed-point table coordinate as the fused kernel
// (spectrum.cu): Q_p is the particle's coordinate, P_b the bin's, and
// f(T) = c0[T >> F] + c1[T >> F] (T mod 2^F) is piecewise linear with its
// kinks where T is a multiple of 2^F (F fraction bits per table segment: 30 here,
// 8 more than the fused kernel's 32-bit coordinate, because the log-linear
// lerp of the steep high-x tail of F magnifies a coordinate's rounding up to a
// thousandfold).  Write R = Pmax - Q (Pmax: the largest bin coordinate of the
// slice) and D_b = Pmax - P_b, so T = R - D_b, and split both into a cell (bits F
// and up) and a low part: R = (Rc, Rl), D_b = (Dc_b, Dl_b).  Then the segment of
// (p, b) is Rc - Dc_b when Rl >= Dl_b and Rc - Dc_b - 1 otherwise, and the
// position inside it is Rl - Dl_b (+ 2^F).  So within an
// interval of R that lies in one cell and between two consecutive low parts
// Dl of the slice's bins, every bin's f is one linear function of Rl, and the
// sums over the particles in that interval need only
//     M0 = sum A_p,   M1 = sum A_p Rl_p.
// The deposit kernel computes each particle's (Q, A) once (pair_stage.cuh), finds
// its interval (cell, rank of Rl among the sorted Dl) and adds (A, A Rl) to
// that interval's FP64 moments; the finish kernel forms each cell row's sums below and
// above every threshold and sums, for every bin, over the at most 200 cells its table
// segments reach:
//     S_b / e_b = sum_cells c0[s] U0 + c1[s] (U1 - Dl_b U0)
//                         + c0[s-1] L0 + c1[s-1] (L1 - (Dl_b - 2^F) L0),
// s = Rc - Dc_b, L = moments of the cell's intervals below Dl_b, U = the rest.
// The work is one particle stage per particle plus (cells x bins), not
// (particles x bins), and the per-(particle, bin) value of f is summed exactly
// (FP64 moments, double-float sums over them) instead of being rounded to FP32 per eval.
// The FP64 atomic sums make the result independent of the particle order up to
// FP64 rounding, not bit for bit.
#include "pair_stage.cuh"

#include <algorithm>
#include <cmath>
#include <cstring>
#include <limits>
#include <numeric>
#include <type_traits>
#include <vector>

namespace rg {

  namespace {

    constexpr int kMomFrac       = kFrac + 8;        // fraction bits of the coordinate
    constexpr int kMomExtra      = 8;                // bits below them before rounding (LogParams::fx)
    constexpr int kMomBuckets    = 4096;             // buckets over the low kMomFrac bits
    constexpr int kMomBucketBits = kMomFrac - 12;
    constexpr int kMomSharedSeg  = kPairSharedSeg;   // largest run in segments
    constexpr int kMomBlocksPerSM = 2;
    constexpr int kMomMaxTable   = 256;              // largest reference table (segments) this path takes
    constexpr size_t kMomMaxBytes = size_t(8) << 30; // histogram memory above which the fused kernel runs

    struct MomentParams {
      FusedParams     fp;      // kinematics constants, status
      LogParams       log;
      const int64_t*  range;   // per slice: (Pmin, Pmax) in kMomFrac units
      int64_t         L;       // table segments << kMomFrac
      PairStreams     in;
      const int4*     mslice;  // per slice: (valid bins, cells, histogram offset, 0)
      const int32_t*  thr;     // per slice: kSliceBins sorted low parts
      const uint32_t* bucket;  // per slice: kMomBuckets entries (bucket_entry)
      double*         hist;    // nseg x per_seg interval moments (M0, M1)
      int64_t         per_seg;
      RunSums         run;
    };

    // A bucket's entry: with `first` thresholds below the bucket and at most one inside it, at
    // offset t (2^kMomBucketBits: none), (entry + offset of Rl) >> kMomBucketBits is the rank of
    // Rl.  With more thresholds inside: bit 31, first << 10 and their count, for a search.
    uint32_t bucket_entry(int first, int count, int64_t t) {
      if (count > 1) {
        return 0x80000000u | (static_cast<uint32_t>(first) << 10) | static_cast<uint32_t>(count);
      }
      const uint32_t width = 1u << kMomBucketBits;
      return static_cast<uint32_t>(first) * width + (count ? width - static_cast<uint32_t>(t) : 0u);
    }

    // The rank of Rl from its bucket's entry when the bucket holds more than one threshold.
    __device__ __noinline__ uint32_t rank_search(uint32_t e, uint32_t Rl, const int32_t* thr) {
      uint32_t lo = (e >> 10) & 0x3ffu, hi = lo + (e & 0x3ffu);
      while (lo < hi) {
        const uint32_t mid = (lo + hi) >> 1;
        if (static_cast<uint32_t>(__ldg(thr + mid)) <= Rl) {
          lo = mid + 1;
        } else {
          hi = mid;
        }
      }
      return lo;
    }

    // Adds (M0, M1) = (A, A Rl) of every lane's particle (idx: its entry, kNoEntry for none) to the
    // moment table.  The L2 takes one request per 32-byte sector and instruction, so the two
    // lanes of a pair add both halves of one particle's entry in one instruction, then both
    // halves of the other's: 1.95e11 particles/s, against 1.0e11 when each lane adds its own two
    // halves in turn (measured on random entries of a 4.3 MB table).  Called by whole warps.
    __device__ __forceinline__ void red_pair(double* hist, uint32_t idx, float A, uint32_t Rl) {
      const bool   odd = threadIdx.x & 1;
      const double M0  = static_cast<double>(A);
      // A Rl = A (2^52 + Rl) - A 2^52, one rounding: the integer enters by its bits
      const double K   = __hiloint2double(0x43300000, static_cast<int>(Rl));
      const double nAK = __hiloint2double((__double2hiint(M0) + 0x03400000) ^ 0x80000000, __double2loint(M0));
      const double M1  = fma(M0, K, nAK);
      const double recv  = __shfl_xor_sync(0xffffffffu, odd ? M0 : M1, 1);
      const uint32_t oth = __shfl_xor_sync(0xffffffffu, idx, 1);
      const uint32_t ia = odd ? oth : idx, ib = odd ? idx : oth;
      double* half = hist + (threadIdx.x & 1);
      red_add_if(ia != kNoEntry, half + 2 * static_cast<size_t>(ia), odd ? recv : M0);
      red_add_if(ib != kNoEntry, half + 2 * static_cast<size_t>(ib), odd ? M1 : recv);
    }

    // Two particles per thread and step (256 apart, so every load is coalesced whatever the
    // streams' alignment), in kSets register sets in turn: a step's loads are issued kSets - 1
    // steps ahead, because they queue behind the reductions in the load-store path (over 2 us),
    // and need no copies between registers.  28 B per particle (u, B, w).  The grid is what fits
    // at once.  Indices are 32-bit within the launch's window of at most 2^31 particles; streams
    // that are not given read a constant with a stride of 0, so the loads carry no tests.
    // Measured on 9.9e7 dump particles x 512 bins: 0.89 ms in two launches (1.11e11 particles/s,
    // 3.1 TB/s) against 1.45 ms for one particle per thread with scalar double-floats, 444
    // instructions a particle and two reduction requests; now 171 and one.  Without the
    // reductions it would take 0.65 ms, the reductions alone 0.69 ms: the L2's reduction requests
    // and the loads behind them set its pace.  Also measured: three blocks per SM 0.95 ms, loads
    // staged through shared memory by cp.async 0.93 ms, entries scattered over the table no gain.
    template <bool kE, bool kSeg>
    __global__ void __launch_bounds__(kPairThreads, kMomBlocksPerSM)
      moments_deposit_kernel(const __grid_constant__ MomentParams m) {
      __shared__ __align__(16) uint32_t bucket[kMomBuckets]; // staged 16 bytes at a time
      __shared__ int64_t                logt[kLogEntries];
      __shared__ uint32_t               soff[kSeg ? kMomSharedSeg + 1 : 1];
      clear_run_sums(m.run);
      const int  slice = blockIdx.y;
      const int4 ms    = m.mslice[slice];
      stage_log_table(m.log, kMomExtra, m.range[2 * slice + 1], logt, kPairThreads);
      for (int i = threadIdx.x; i < kMomBuckets / 4; i += kPairThreads) {
        reinterpret_cast<uint4*>(bucket)[i] = reinterpret_cast<const uint4*>(m.bucket + slice * kMomBuckets)[i];
      }
      if (!stage_segments<kSeg>(m.in, m.fp.status, soff)) {
        return;
      }
      const int64_t  Pmin = m.range[2 * slice], Pmax = m.range[2 * slice + 1];
      const uint32_t row = static_cast<uint32_t>(ms.x) + 1u, nc = static_cast<uint32_t>(ms.y);
      const int32_t* thr = m.thr + slice * kSliceBins;
      LogParams      lg  = m.log;
      lg.fx              = kMomExtra;
      const uint32_t first = kSeg ? soff[0] : 0u;
      const uint32_t last  = kSeg ? soff[m.in.nseg] : static_cast<uint32_t>(min(m.in.n - m.in.window, kPairWindow));
      const uint32_t step  = gridDim.x * kPairChunk, tid = threadIdx.x;

      constexpr int kSets = kE ? 2 : 3; // with E a third set spills (64.2 us against 60.5 for 4.3e6 particles)
      uint32_t useg = 0, uend = kSeg ? soff[1] : last; // the segment of the step's first particle, and its end
      auto     add  = [&](uint32_t base, const float2 (&from)[kComps]) {
        f2 v[kComps];
        to_pairs<kE>(from, v);
        const Place2 pl = place2<kE>(v, m.fp, lg, logt, Pmin, Pmax, m.L);
        if (kSeg) {
          while (uend <= base) { // base < last = soff[nseg]
            ++useg;
            uend = soff[useg + 1];
          }
        }
        uint32_t Rl[2], idx[2], e[2], Rc[2];
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          Rc[j]  = static_cast<uint32_t>(static_cast<int32_t>(pl.Y[j] >> 32) >> (kMomFrac + kMomExtra - 32));
          Rl[j]  = static_cast<uint32_t>(pl.Y[j] >> kMomExtra) & ((1u << kMomFrac) - 1u);
          e[j]   = bucket[Rl[j] >> kMomBucketBits];
          idx[j] = (e[j] + (Rl[j] & ((1u << kMomBucketBits) - 1u))) >> kMomBucketBits;
        }
        if ((e[0] | e[1]) & 0x80000000u) {
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            if (e[j] & 0x80000000u) {
              idx[j] = rank_search(e[j], Rl[j], thr);
            }
          }
        }
        const uint32_t origin = static_cast<uint32_t>(ms.z) + (kSeg ? useg * static_cast<uint32_t>(m.per_seg) : 0u);
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          idx[j] += origin + Rc[j] * row;
          idx[j] = Rc[j] < nc && emits(pl.A[j]) ? idx[j] : kNoEntry;
        }
        if (base + kPairChunk > (kSeg ? uend : last)) { // the step crosses an end of its segment or of the particles
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            const uint32_t i = base + tid + j * kPairThreads;
            if (i >= last) {
              idx[j] = kNoEntry;
            } else if (kSeg && idx[j] != kNoEntry) {
              for (uint32_t seg = useg; soff[seg + 1] <= i; ++seg) { // i < soff[nseg]
                idx[j] += static_cast<uint32_t>(m.per_seg);
              }
            }
          }
        }
        __syncwarp();
        red_pair(m.hist, idx[0], pl.A[0], Rl[0]);
        red_pair(m.hist, idx[1], pl.A[1], Rl[1]);
      };
      float2   set[kSets][kComps];
      uint32_t base = first + blockIdx.x * kPairChunk;
#pragma unroll
      for (int k = 0; k < kSets - 1; ++k) {
        load_pair<kE>(m.in, base + k * step, last, set[k]);
      }
      while (base < last) {
#pragma unroll
        for (int k = 0; k < kSets; ++k) {
          load_pair<kE>(m.in, base + (kSets - 1) * step, last, set[(k + kSets - 1) % kSets]);
          add(base, set[k]);
          base += step;
          if (base >= last) {
            break;
          }
        }
      }
    }

    // ---- finish: row sums, then every bin over its cells ------------------------------------
    struct MomentFinishParams {
      double2*        hist;     // read, and set back to zero for the next run
      int64_t         per_seg;
      const int4*     mslice;
      const int4*     bins;     // per slice: kSliceBins (sorted position, cell offset Dc, low part Dl, bin in the
                                // slice) by ascending Dc, the rest with Dc = INT_MAX
      const float4*   coef;     // -1 .. nseg_tab: (c0, c1) as double-floats, c1 per segment; both ends zero
      int             nseg_tab; // table segments
      int             nslices;
      int             nbins;
      const float*    ebins;
      const unsigned* status;
      double*         acc;      // [nseg][nslices][kSliceBins], cleared by the deposit
      unsigned*       done;     // [nseg][nslices] blocks finished, cleared by the deposit
      float*          out;      // nseg x nbins
      f2              nz;       // of product2
    };

    constexpr int kFinWarps = 8;
    constexpr int kFinThreads = 32 * kFinWarps;

    // A bin as the finish kernel reads it: (sorted position, Dc), and -Dl and 1 - Dl in segment
    // units as double-floats.
    struct FinBin {
      int    pos, Dc;
      float  nDh, nDl, mDh, mDl;
    };

    // Shared memory: coefficients, bins, and per warp the bins' sums, the row (overwritten by the
    // sums below) and the sums above.
    size_t finish_smem(int max_bins, int nseg_tab) {
      const size_t row = max_bins + 1, groups = (max_bins + 31) & ~31;
      return sizeof(float4) * (nseg_tab + 2) + sizeof(FinBin) * groups +
             kFinWarps * (sizeof(float2) * groups + sizeof(float4) * 2 * row);
    }

    __device__ __forceinline__ ff2 shfl_up_ff2(ff2 a, int o) {
      return { { __shfl_up_sync(0xffffffffu, a.hi.v, o) }, { __shfl_up_sync(0xffffffffu, a.lo.v, o) } };
    }

    __device__ __forceinline__ ff2 shfl_down_ff2(ff2 a, int o) {
      return { { __shfl_down_sync(0xffffffffu, a.hi.v, o) }, { __shfl_down_sync(0xffffffffu, a.lo.v, o) } };
    }

    __device__ __forceinline__ void store_ff2(float4* to, ff2 a) {
      float4 f;
      unpack2(a.hi, f.x, f.y);
      unpack2(a.lo, f.z, f.w);
      *to = f;
    }

    // The packed sums of a warp hold entries from 2^-kFinBelow to 2^kFinAbove times its scale with all their
    // bits: split_double keeps 2^-44 down to 2^-74 and anything down to 2^-126, and the coefficients are
    // not below 2^-34.  Rows that reach further start a new scale, and a row that spans more by itself
    // (a particle that outweighs a neighbour by 1e18) is summed in FP64.
    constexpr int kFinBelow = 60, kFinAbove = 40;

    // The warp's bin sums into the slice's, in FP64, and back to zero.
    __device__ __noinline__ void flush_sums(float2* acc, int nv, int scale, double* total) {
      const double s = __hiloint2double((scale + 1023) << 20, 0);
      for (int i = threadIdx.x & 31; i < nv; i += 32) {
        const float2 a = acc[i];
        if (a.x != 0.0f) {
          atomicAdd(total + i, (static_cast<double>(a.x) + static_cast<double>(a.y)) * s);
        }
        acc[i] = make_float2(0.0f, 0.0f);
      }
    }

    // A row of cell c in FP64, from its copy in shared memory: sums below in place, sums above beside
    // it, then every bin's share into the slice's sums.
    __device__ __noinline__ void wide_row(double2* row_sums, double2* above, const float4* coef, const FinBin* bins, int nv,
                                          int c, int nseg_tab, double* total) {
      const int lane = threadIdx.x & 31, row = nv + 1, per = (row + 31) / 32;
      const int j0 = min(lane * per, row), j1 = min(j0 + per, row);
      double    l0 = 0.0, l1 = 0.0;
      for (int j = j0; j < j1; ++j) {
        l0 += row_sums[j].x;
        l1 += row_sums[j].y;
      }
      double u0 = l0, u1 = l1;
      for (int o = 1; o < 32; o <<= 1) {
        const double a0 = __shfl_up_sync(0xffffffffu, l0, o), a1 = __shfl_up_sync(0xffffffffu, l1, o);
        const double b0 = __shfl_down_sync(0xffffffffu, u0, o), b1 = __shfl_down_sync(0xffffffffu, u1, o);
        if (lane >= o) {
          l0 += a0;
          l1 += a1;
        }
        if (lane + o < 32) {
          u0 += b0;
          u1 += b1;
        }
      }
      l0 = __shfl_up_sync(0xffffffffu, l0, 1);
      l1 = __shfl_up_sync(0xffffffffu, l1, 1);
      u0 = __shfl_down_sync(0xffffffffu, u0, 1);
      u1 = __shfl_down_sync(0xffffffffu, u1, 1);
      if (lane == 0) {
        l0 = l1 = 0.0;
      }
      if (lane == 31) {
        u0 = u1 = 0.0;
      }
      for (int j = j1 - 1; j >= j0; --j) {
        above[j] = make_double2(u0, u1);
        u0 += row_sums[j].x;
        u1 += row_sums[j].y;
      }
      for (int j = j0; j < j1; ++j) {
        l0 += row_sums[j].x;
        l1 += row_sums[j].y;
        row_sums[j] = make_double2(l0, l1);
      }
      __syncwarp();
      const double unit = 1.0 / (1u << kMomFrac);
      for (int i = lane; i < nv; i += 32) {
        const FinBin b = bins[i];
        const int    s = c - b.Dc;
        if (s >= 0 && s <= nseg_tab) {
          const float4  ku = coef[s + 1], kl = coef[s];
          const double2 U = above[b.pos], L = row_sums[b.pos];
          const double  nD = static_cast<double>(b.nDh) + static_cast<double>(b.nDl);
          const double  mD = static_cast<double>(b.mDh) + static_cast<double>(b.mDl);
          const double  y  = (static_cast<double>(ku.x) + static_cast<double>(ku.y)) * U.x +
                           (static_cast<double>(ku.z) + static_cast<double>(ku.w)) * (U.y * unit + nD * U.x) +
                           (static_cast<double>(kl.x) + static_cast<double>(kl.y)) * L.x +
                           (static_cast<double>(kl.z) + static_cast<double>(kl.w)) * (L.y * unit + mD * L.x);
          if (y != 0.0) {
            atomicAdd(total + i, y);
          }
        }
      }
      __syncwarp(); // the row's buffer takes the next row
    }

    // One warp per cell row, kFinWarps rows in flight per block, blockIdx.y = (segment, slice).
    // The row is copied to shared memory (coalesced) and set back to zero; a lane takes C consecutive
    // entries (M0, and M1 in segment units, as packed double-floats scaled by a power of two), and the
    // warp leaves the row's sums below (L) and above (U) every threshold in shared memory.  U is summed from the row's end, not as
    // total - L, so that a bin with no particle above its threshold gets an exact zero.  Then
    // lanes own bins in the order of their cells, so that whole groups of 32 skip the cells their
    // table segments do not reach.  Double-floats (2^-44) because the FP64 pipe issues 1.6
    // operations per clock and SM: the FP64 scan and reduce kernels this replaces took 503 and
    // 449 us for 256 spectra of 200 bins (this kernel 124 us, and no memset of 350 MB before the
    // run).  What bounds it is the latency of its chains: rows fetched one ahead take a third buffer, and
    // with it two blocks fit an SM (146 us) instead of three; the launch bounds keep the registers to
    // that.  Blocks add their bins' sums in FP64; the last block of a (segment, slice) writes the spectrum.
    template <int C>
    __global__ void __launch_bounds__(kFinThreads, C <= 4 ? 4 : C <= 8 ? 3 : C <= 12 ? 2 : 1) moments_finish_kernel(const __grid_constant__ MomentFinishParams r) {
      extern __shared__ __align__(16) unsigned char smem[];
      __shared__ int   wscale[kFinWarps];
      __shared__ bool  last;
      const int  seg = blockIdx.y / r.nslices, slice = blockIdx.y % r.nslices;
      const int4 ms  = r.mslice[slice];
      const int  nv = ms.x, row = nv + 1, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
      const int  groups = (nv + 31) & ~31; // bins in groups of 32
      float4*    coef  = reinterpret_cast<float4*>(smem);
      FinBin*    bins  = reinterpret_cast<FinBin*>(coef + r.nseg_tab + 2);
      float2*    sums  = reinterpret_cast<float2*>(bins + groups); // [kFinWarps][groups]
      float2*    acc   = sums + warp * groups;
      float4*    buf   = reinterpret_cast<float4*>(sums + kFinWarps * groups) + 2 * warp * row;
      float4*    Us    = buf + row;
      double2*   hist  = r.hist + seg * r.per_seg + ms.z;
      double*    total = r.acc + static_cast<int64_t>(blockIdx.y) * kSliceBins;
      const int  c0 = blockIdx.x * kFinWarps + warp, cstep = gridDim.x * kFinWarps;
      auto fetch = [&](int c) {
        if (c < ms.y) {
          double2* h = hist + static_cast<int64_t>(c) * row;
          for (int j = lane; j < row; j += 32) {
            copy16(smem_u32(buf + j), h + j);
          }
        }
        copies_commit();
      };
      fetch(c0);
      const bool failed = *r.status != kDevOk;
      for (int i = threadIdx.x; i < r.nseg_tab + 2; i += kFinThreads) {
        coef[i] = r.coef[i];
      }
      for (int i = threadIdx.x; i < groups; i += kFinThreads) {
        const int4  b  = r.bins[slice * kSliceBins + i];
        const float un = 1.0f / (1u << kMomFrac);
        const int   m  = (1 << kMomFrac) - b.z;
        const float dh = static_cast<float>(b.z), mh = static_cast<float>(m);
        bins[i] = FinBin { b.x, b.y, -dh * un, static_cast<float>(static_cast<int>(dh) - b.z) * un, mh * un,
                           static_cast<float>(m - static_cast<int>(mh)) * un };
      }
      for (int i = lane; i < groups; i += 32) {
        acc[i] = make_float2(0.0f, 0.0f);
      }
      __syncthreads();
      int scale = -2000; // this warp's sums hold their value times 2^-scale
#pragma unroll 1
      for (int c = c0; c < ms.y; c += cstep) {
        if (c != c0) {
          fetch(c);
        }
        copies_wait<0>();
        __syncwarp(); // every lane's copies of this row have landed
        double2* h = hist + static_cast<int64_t>(c) * row;
        double2  d[C];
        int      top = 0, low = 0x7ff; // largest and smallest exponent of the row
#pragma unroll
        for (int k = 0; k < C; ++k) {
          const int j = lane * C + k;
          d[k]        = j < row ? *reinterpret_cast<const double2*>(buf + j) : make_double2(0.0, 0.0);
          const int e0 = (__double2hiint(d[k].x) >> 20) & 0x7ff, e1 = ((__double2hiint(d[k].y) >> 20) & 0x7ff) - kMomFrac;
          top = max(top, max(e0, e1));
          low = min(low, e0 > 0 ? e0 : e1 > 0 ? e1 : 0x7ff); // of M0; M1 matters beside it only as much as it is large
        }
        top = __reduce_max_sync(0xffffffffu, top);
        low = __reduce_min_sync(0xffffffffu, low);
        if (top == 0) { // an empty row
          continue;
        }
        for (int j = lane; j < row; j += 32) {
          h[j] = make_double2(0.0, 0.0);
        }
        if (failed) {
          continue;
        }
        if (top - low > kFinBelow) {
          __syncwarp(); // every lane has read the row
          wide_row(reinterpret_cast<double2*>(buf), reinterpret_cast<double2*>(Us), coef, bins, nv, c, r.nseg_tab, total);
          continue;
        }
        if (top - 1023 > scale + kFinAbove || low - 1023 < scale - kFinBelow) {
          if (scale > -2000) {
            flush_sums(acc, nv, scale, total);
          }
          scale = top - 1023;
        }
        ff2 v[C];
        ff2 t { set2(0.0f), set2(0.0f) };
#pragma unroll
        for (int k = 0; k < C; ++k) {
          const float2 m0 = split_double(d[k].x, scale), m1 = split_double(d[k].y, scale + kMomFrac);
          v[k]            = ff2 { pack2(m0.x, m1.x), pack2(m0.y, m1.y) };
          t               = ff_add2(t, v[k]);
        }
        // exclusive sums of the lanes below and above
        ff2 lo = t, up = t;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const ff2 a = shfl_up_ff2(lo, o), b = shfl_down_ff2(up, o);
          if (lane >= o) {
            lo = ff_add2(a, lo);
          }
          if (lane + o < 32) {
            up = ff_add2(up, b);
          }
        }
        lo = shfl_up_ff2(lo, 1);
        up = shfl_down_ff2(up, 1);
        if (lane == 0) {
          lo = ff2 { set2(0.0f), set2(0.0f) };
        }
        if (lane == 31) {
          up = ff2 { set2(0.0f), set2(0.0f) };
        }
        __syncwarp(); // the row is in registers: its buffer takes the sums below
#pragma unroll
        for (int k = 0; k < C; ++k) {
          lo           = ff_add2(lo, v[k]);
          const int kr = C - 1 - k;
          if (lane * C + k < row) {
            store_ff2(buf + lane * C + k, lo);
          }
          if (lane * C + kr < row) {
            store_ff2(Us + lane * C + kr, up);
          }
          up = ff_add2(v[kr], up);
        }
        __syncwarp();
#pragma unroll 1
        for (int q = 0; q < nv; q += 32) {
          if (c < bins[q].Dc || c > bins[min(q + 31, nv - 1)].Dc + r.nseg_tab) { // warp-uniform
            continue;
          }
          const FinBin b = bins[q + lane];
          const int    s = c - b.Dc;
          if (s >= 0 && s <= r.nseg_tab) {
            const float4 ku = coef[s + 1], kl = coef[s]; // segments s and s - 1
            const float4 U = Us[b.pos], Lo = buf[b.pos];
            // pairs (U, L): x = M1 - (Dl, Dl - 1) M0, then c0 M0 + c1 x
            const ff2 M0 { pack2(U.x, Lo.x), pack2(U.z, Lo.z) }, M1 { pack2(U.y, Lo.y), pack2(U.w, Lo.w) };
            const ff2 x = ff_add2(M1, ff_mul2(ff2 { pack2(b.nDh, b.mDh), pack2(b.nDl, b.mDl) }, M0, r.nz));
            const ff2 k0 { pack2(ku.x, kl.x), pack2(ku.y, kl.y) }, k1 { pack2(ku.z, kl.z), pack2(ku.w, kl.w) };
            const ff2 y = ff_add2(ff_mul2(k0, M0, r.nz), ff_mul2(k1, x, r.nz));
            float     h0, h1, l0, l1;
            unpack2(y.hi, h0, h1);
            unpack2(y.lo, l0, l1);
            const float2 a = acc[q + lane];
            const ff     n = ff_add(ff { a.x, a.y }, ff_add(ff { h0, l0 }, ff { h1, l1 }));
            acc[q + lane]  = make_float2(n.hi, n.lo);
          }
        }
        __syncwarp(); // the row's buffer takes the next row
      }
      copies_wait<0>();
      // the block's sums, at its warps' largest scale, one FP64 add per bin
      if (lane == 0) {
        wscale[warp] = scale;
      }
      __syncthreads();
      int top = wscale[0];
#pragma unroll
      for (int w = 1; w < kFinWarps; ++w) {
        top = max(top, wscale[w]);
      }
      if (top > -2000) {
        const double s2 = __hiloint2double((top + 1023) << 20, 0);
        for (int i = threadIdx.x; i < nv; i += kFinThreads) {
          ff     t { 0.0f, 0.0f };
          double far = 0.0; // of warps whose scale is too far below for the packed sum
#pragma unroll
          for (int w = 0; w < kFinWarps; ++w) {
            const int    down = top - wscale[w];
            const float2 a    = sums[w * groups + i];
            if (down <= kFinAbove) {
              const float f = __uint_as_float(static_cast<uint32_t>(127 - down) << 23);
              t             = ff_add(t, ff { a.x * f, a.y * f });
            } else if (a.x != 0.0f) {
              far += (static_cast<double>(a.x) + static_cast<double>(a.y)) * __hiloint2double((wscale[w] + 1023) << 20, 0);
            }
          }
          if (t.hi != 0.0f || far != 0.0) {
            atomicAdd(total + i, (static_cast<double>(t.hi) + static_cast<double>(t.lo)) * s2 + far);
          }
        }
      }
      __threadfence();
      __syncthreads();
      if (threadIdx.x == 0) {
        last = atomicAdd(r.done + blockIdx.y, 1u) == gridDim.x - 1;
      }
      __syncthreads();
      if (!last) {
        return;
      }
      __threadfence();
      const int   n0   = slice * kSliceBins;
      float*      out  = r.out + static_cast<int64_t>(seg) * r.nbins + n0;
      const float none = failed ? __int_as_float(0x7fffffff) : 0.0f;
      if (failed || nv < min(kSliceBins, r.nbins - n0)) { // bins without a valid energy stay 0
        for (int i = threadIdx.x; i < min(kSliceBins, r.nbins - n0); i += kFinThreads) {
          out[i] = none;
        }
        __syncthreads();
      }
      for (int i = threadIdx.x; i < nv; i += kFinThreads) {
        const double t = __ldcg(total + i);
        const int    j = r.bins[slice * kSliceBins + i].w;
        if (!failed) {
          out[j] = __double2float_rn(t * static_cast<double>(r.ebins[n0 + j]));
        }
      }
    }

    int max_cells(const rg_spectrum_plan* pl) {
      int m = 1;
      for (int s = 0; s < pl->nslices; ++s) {
        m = std::max(m, pl->h_mslice[4 * s + 1]);
      }
      return m;
    }

    int max_valid(const rg_spectrum_plan* pl) {
      int m = 0;
      for (int s = 0; s < pl->nslices; ++s) {
        m = std::max(m, pl->h_mslice[4 * s]);
      }
      return m;
    }

  } // namespace

  // Interval tables of a reference-table particle plan: the bins' coordinates in
  // kMomFrac units (FP64 on the host, as the fused kernel's in kFrac units), their
  // validity, and the table geometry (ln xmin, dln) and ln K0 the coordinates use.
  int moments_prepare(rg_spectrum_plan* pl, const std::vector<uint8_t>& valid, double ln_xmin, double dln,
                      double ln_k0) {
    pl->moments_ok = false;
    if (pl->table_mode == kModeSmooth && pl->aligned) {
      return smooth_moments_prepare(pl, ln_k0);
    }
    if (pl->table_mode != kModeRef || pl->source != kSrcParticles || pl->ref->n - 1 > kMomMaxTable) {
      return RG_OK;
    }
    const int            ns    = pl->nslices;
    const double         scale = std::ldexp(1.0, kMomFrac) / dln;
    const int64_t        L     = static_cast<int64_t>(pl->ref->n - 1) << kMomFrac;
    const int64_t        mask  = (int64_t(1) << kMomFrac) - 1;
    std::vector<int64_t> Ps(std::max(pl->nbins, 1), 0);
    std::vector<int64_t> range(2 * static_cast<size_t>(ns), 0);
    std::vector<int32_t> thr(static_cast<size_t>(ns) * kSliceBins, 0);
    std::vector<uint32_t> bucket(static_cast<size_t>(ns) * kMomBuckets, 0);
    std::vector<int4>    binfo(static_cast<size_t>(ns) * kSliceBins,
                               make_int4(0, std::numeric_limits<int>::max(), 0, 0));
    pl->h_mslice.assign(4 * static_cast<size_t>(ns), 0);
    int64_t off = 0;
    for (int s = 0; s < ns; ++s) {
      std::vector<int> idx;
      int64_t          Pmin = std::numeric_limits<int64_t>::max(), Pmax = std::numeric_limits<int64_t>::min();
      for (int j = 0; j < kSliceBins; ++j) {
        const int b = s * kSliceBins + j;
        if (b < pl->nbins && valid[b]) {
          Ps[b] = std::llround((std::log(static_cast<double>(pl->h_bins[b])) - ln_xmin - ln_k0) * scale);
          Pmin  = std::min(Pmin, Ps[b]);
          Pmax  = std::max(Pmax, Ps[b]);
          idx.push_back(b);
        }
      }
      if (idx.empty()) {
        Pmin = Pmax = 0;
      }
      range[2 * s]     = Pmin;
      range[2 * s + 1] = Pmax;
      const auto low = [&](int b) { return static_cast<int32_t>((Pmax - Ps[b]) & mask); };
      std::stable_sort(idx.begin(), idx.end(), [&](int a, int b) { return low(a) < low(b); });
      const int nv = static_cast<int>(idx.size());
      int4*     bi = binfo.data() + static_cast<size_t>(s) * kSliceBins;
      for (int k = 0; k < nv; ++k) {
        const int b = idx[k];
        thr[static_cast<size_t>(s) * kSliceBins + k] = low(b);
        bi[k] = make_int4(k, static_cast<int>((Pmax - Ps[b]) >> kMomFrac), low(b), b - s * kSliceBins);
      }
      std::stable_sort(bi, bi + nv, [](const int4& x, const int4& y) { return x.y < y.y; });
      for (int k = 0, c = 0; k < kMomBuckets; ++k) {
        const int64_t  edge = static_cast<int64_t>(k) << kMomBucketBits, end = edge + (int64_t(1) << kMomBucketBits);
        const int32_t* t    = thr.data() + static_cast<size_t>(s) * kSliceBins;
        const int      c0   = c;
        while (c < nv && t[c] < end) {
          ++c;
        }
        bucket[static_cast<size_t>(s) * kMomBuckets + k] = bucket_entry(c0, c - c0, c > c0 ? t[c0] - edge : 0);
      }
      // live particles have Pmax - Q in [0, Pmax - Pmin + L)
      const int64_t cells = nv ? ((Pmax - Pmin + L - 1) >> kMomFrac) + 1 : 1;
      if (off + cells * (nv + 1) > std::numeric_limits<int32_t>::max()) {
        return RG_OK; // too large for this path; the fused kernel serves the plan
      }
      pl->h_mslice[4 * s + 0] = nv;
      pl->h_mslice[4 * s + 1] = static_cast<int32_t>(cells);
      pl->h_mslice[4 * s + 2] = static_cast<int32_t>(off);
      off += cells * (nv + 1);
    }
    pl->hist_per_seg = off;
    pl->mom_L        = L;
    // segment coefficients of the reference's log-linear lerp (tabulation.hpp:39-41) in the
    // ideal coordinate, F = c0 + c1 (position in the segment), as double-floats; entry i + 1 is
    // segment i, the ends are zero
    const int           nt = pl->ref->n - 1;
    std::vector<float4> coef(nt + 2, make_float4(0.0f, 0.0f, 0.0f, 0.0f));
    const double        d10 = pl->ref->dln / M_LN10;
    for (int i = 0; i < nt; ++i) {
      const double xa = pl->ref->h_x[i], xb = pl->ref->h_x[i + 1], ya = pl->ref->h_y[i], yb = pl->ref->h_y[i + 1];
      const double beta = (yb - ya) / std::log10(xb / xa);
      const double c0   = ya + beta * (pl->ref->ln_xmin / M_LN10 + i * d10 - std::log10(xa));
      const double c1   = beta * d10;
      const float  h0 = static_cast<float>(c0), h1 = static_cast<float>(c1);
      coef[i + 1]     = make_float4(h0, static_cast<float>(c0 - h0), h1, static_cast<float>(c1 - h1));
    }
    RG_TRY(fixed_log_prepare(pl, kMomFrac, dln));
    if (pl->log_fx != kMomExtra) {
      return RG_OK; // a table spacing the deposit's fixed shifts do not fit; the fused kernel serves the plan
    }
    RG_CUDA_TRY(cudaMalloc(&pl->d_mslice, sizeof(int32_t) * pl->h_mslice.size()));
    RG_CUDA_TRY(cudaMalloc(&pl->d_mrange, sizeof(int64_t) * range.size()));
    RG_CUDA_TRY(cudaMalloc(&pl->d_thr, sizeof(int32_t) * thr.size()));
    RG_CUDA_TRY(cudaMalloc(&pl->d_bucket, sizeof(uint32_t) * bucket.size()));
    RG_CUDA_TRY(cudaMalloc(&pl->d_binfo, sizeof(int4) * binfo.size()));
    RG_CUDA_TRY(cudaMalloc(&pl->d_mcoef, sizeof(float4) * coef.size()));
    RG_CUDA_TRY(cudaMemcpy(pl->d_mslice, pl->h_mslice.data(), sizeof(int32_t) * pl->h_mslice.size(),
                           cudaMemcpyHostToDevice));
    RG_CUDA_TRY(cudaMemcpy(pl->d_mrange, range.data(), sizeof(int64_t) * range.size(), cudaMemcpyHostToDevice));
    RG_CUDA_TRY(cudaMemcpy(pl->d_thr, thr.data(), sizeof(int32_t) * thr.size(), cudaMemcpyHostToDevice));
    RG_CUDA_TRY(cudaMemcpy(pl->d_bucket, bucket.data(), sizeof(uint32_t) * bucket.size(), cudaMemcpyHostToDevice));
    RG_CUDA_TRY(cudaMemcpy(pl->d_binfo, binfo.data(), sizeof(int4) * binfo.size(), cudaMemcpyHostToDevice));
    RG_CUDA_TRY(cudaMemcpy(pl->d_mcoef, coef.data(), sizeof(float4) * coef.size(), cudaMemcpyHostToDevice));
    pl->moments_ok = true;
    return RG_OK;
  }

  // The coordinate's fixed-point constants and log table (pair_stage.cuh) for F fraction bits
  // and node spacing dln; log_fx = 0 where no spacing of units fits (never for these tables).
  int fixed_log_prepare(rg_spectrum_plan* pl, int F, double dln) {
    int fx = 8;
    while (fx > 0 && std::ldexp(1.0, F + fx) / (2.0 * dln) >= std::ldexp(1.0, 40) * 1.8) {
      --fx; // S 2^-10 stays below 1.8 x 2^30
    }
    pl->log_fx = fx;
    if (fx < 1) {
      return RG_OK;
    }
    const double S = std::ldexp(1.0, F + fx) / (2.0 * dln);
    pl->log_Sh     = static_cast<float>(S);
    pl->log_Sl     = static_cast<float>(S - static_cast<double>(pl->log_Sh));
    pl->log_Cfx    = std::llround(S * M_LN2);
    std::vector<int64_t> t(kLogEntries + kStandIn);
    for (int i = 0; i < kLogEntries; ++i) {
      // [0.5, 1), then 1, then [0.25, 0.5) of which only the last entry is ever read
      const double mant = 1.0 + std::ldexp(static_cast<double>(i & 1023), -10);
      t[i]              = std::llround(S * std::log(i < 1024 ? 0.5 * mant : (i == 1024 ? 1.0 : 0.25 * mant)));
    }
    std::vector<float> constants(2 * kStandIn, 0.0f);
    std::fill(constants.begin() + kStandIn, constants.end(), 1.0f);
    std::memcpy(&t[kLogEntries], constants.data(), sizeof(float) * constants.size());
    RG_CUDA_TRY(cudaMalloc(&pl->d_logt, sizeof(int64_t) * t.size()));
    RG_CUDA_TRY(cudaMemcpy(pl->d_logt, t.data(), sizeof(int64_t) * t.size(), cudaMemcpyHostToDevice));
    return RG_OK;
  }

  // Whether a run over nseg segments takes the interval-moment path.
  bool moments_selected(const rg_spectrum_plan* pl, int nseg) {
    if (!pl->moments_ok || pl->algo == RG_ALGO_DIRECT || nseg > kMomSharedSeg) {
      return false;
    }
    return static_cast<size_t>(nseg) * static_cast<size_t>(pl->hist_per_seg) * sizeof(double2) <= kMomMaxBytes;
  }

  // Moment tables and sums for nseg segments.  The tables are zero between runs: zeroed after they are
  // allocated (moments_clear), and by each run's finish kernel, which reads every entry anyway (a memset
  // per run costs a launch for one spectrum, and a pass over 350 MB for 256).  Runs that overlapped (which a
  // plan does not allow) leave them zero too: the finish that starts last comes after all deposits and
  // clears what it finds.
  int moments_reserve(rg_spectrum_plan* pl, int nseg) {
    const size_t need = static_cast<size_t>(nseg) * static_cast<size_t>(pl->hist_per_seg);
    if (need > pl->hist_cap) {
      cudaFree(pl->d_hist);
      pl->d_hist   = nullptr;
      pl->hist_cap = 0;
      RG_CUDA_TRY(cudaMalloc(&pl->d_hist, sizeof(double2) * need));
      pl->hist_cap   = need;
      pl->hist_dirty = true; // not zero yet
    }
    const size_t sums = static_cast<size_t>(nseg) * pl->nslices;
    if (sums > pl->msum_cap) {
      cudaFree(pl->d_msum);
      pl->d_msum   = nullptr;
      pl->msum_cap = 0;
      const size_t bytes = sums * (sizeof(double) * kSliceBins + sizeof(unsigned));
      RG_CUDA_TRY(cudaMalloc(&pl->d_msum, bytes)); // cleared by each run
      pl->msum_cap = sums;
    }
    return RG_OK;
  }

  // The tables zero, as of the work queued on s before this call.
  int moments_clear(rg_spectrum_plan* pl, cudaStream_t s) {
    if (pl->hist_dirty) {
      RG_CUDA_TRY(cudaMemsetAsync(pl->d_hist, 0, sizeof(double2) * pl->hist_cap, s));
      pl->hist_dirty = false;
    }
    return RG_OK;
  }

  // Before a run's deposits: the tables of nseg segments, zero (also new ones, and after a run that
  // failed between its deposit and its finish).  A captured run only records its memset and its
  // finish: tables that were not zero before it are still not zero for the next run that executes.
  int moments_begin(rg_spectrum_plan* pl, int nseg, cudaStream_t s) {
    RG_TRY(moments_reserve(pl, nseg));
    bool recorded = false;
    if (pl->hist_dirty) {
      cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
      RG_CUDA_TRY(cudaStreamIsCapturing(s, &capture));
      recorded = capture != cudaStreamCaptureStatusNone;
    }
    RG_TRY(moments_clear(pl, s));
    pl->hist_dirty       = true;
    pl->hist_stays_dirty = recorded;
    return RG_OK;
  }

  // A run without particles has no deposit.
  int moments_clear_sums(rg_spectrum_plan* pl, cudaStream_t s) {
    const RunSums r = run_sums(pl, 1);
    RG_CUDA_TRY(cudaMemsetAsync(r.sums, 0, sizeof(double) * r.nsums, s));
    RG_CUDA_TRY(cudaMemsetAsync(r.done, 0, sizeof(unsigned) * r.ndone, s));
    return RG_OK;
  }

  int moments_deposit(rg_spectrum_plan* pl, const float* const comp[kComps], const int64_t* d_off, int64_t n,
                      int nseg, cudaStream_t s) {
    if (pl->aligned) {
      return smooth_moments_deposit(pl, comp, d_off, n, nseg, s);
    }
    MomentParams m {};
    fill_params(pl, comp, nullptr, nullptr, n, 1, m.fp);
    m.range   = pl->d_mrange;
    m.L       = pl->mom_L;
    m.mslice  = reinterpret_cast<const int4*>(pl->d_mslice);
    m.thr     = pl->d_thr;
    m.bucket  = pl->d_bucket;
    m.hist    = reinterpret_cast<double*>(pl->d_hist);
    m.per_seg = pl->hist_per_seg;
    m.run     = run_sums(pl, d_off ? nseg : 1);
    fill_log_params(pl, m.log);
    DeviceContext* ctx = nullptr;
    RG_TRY(context(&ctx));
    if (n == 0 && !d_off) {
      return moments_clear_sums(pl, s);
    }
    std::pair<cudaEvent_t, cudaEvent_t> ev { nullptr, nullptr };
    if (pl->timing) {
      if (pl->ev_free.empty()) {
        RG_CUDA_TRY(cudaEventCreate(&ev.first));
        RG_CUDA_TRY(cudaEventCreate(&ev.second));
      } else {
        ev = pl->ev_free.back();
        pl->ev_free.pop_back();
      }
      RG_CUDA_TRY(cudaEventRecord(ev.first, s));
    }
    for (int64_t w = 0; w < std::max<int64_t>(n, 1); w += kPairWindow) {
      fill_streams(pl, comp, d_off, n, nseg, w, m.in);
      const dim3 blocks(pair_grid(n, w, ctx->sms, kMomBlocksPerSM), pl->nslices);
      if (m.fp.has_e) {
        if (d_off) {
          moments_deposit_kernel<true, true><<<blocks, kPairThreads, 0, s>>>(m);
        } else {
          moments_deposit_kernel<true, false><<<blocks, kPairThreads, 0, s>>>(m);
        }
      } else if (d_off) {
        moments_deposit_kernel<false, true><<<blocks, kPairThreads, 0, s>>>(m);
      } else {
        moments_deposit_kernel<false, false><<<blocks, kPairThreads, 0, s>>>(m);
      }
    }
    RG_CUDA_TRY(cudaGetLastError());
    if (pl->timing) {
      RG_CUDA_TRY(cudaEventRecord(ev.second, s));
      pl->ev_used.push_back(ev);
    }
    return RG_OK;
  }

  namespace {

    // Blocks per (segment, slice): those with which the waves of `resident` blocks take the fewest rows
    // of a warp, a block's setup and epilogue counted as kFinSetup rows.  Runs of few particles (counted as
    // 0 / 1 / 3 rows): 256 spectra x 200 bins 193 / 122 / 128 us, 256 x 512 641 / 368 / 354, 1024 x 100 485 /
    // 258 / 257, 16 x 512 66 / 44 / 44; from one to four spectra, and 64 x 200, the same with all three.
    constexpr size_t kFinSmSmem = 227 * 1024;
    constexpr int    kFinSetup  = 1;
    int finish_blocks(int rows, int cells, int resident) {
      const int most = std::max(1, (cells + kFinWarps - 1) / kFinWarps);
      int       best = 1;
      int64_t   least = std::numeric_limits<int64_t>::max();
      for (int gx = 1; gx <= most; ++gx) {
        const int64_t waves = (static_cast<int64_t>(rows) * gx + resident - 1) / resident;
        const int64_t cost  = waves * ((cells + kFinWarps * gx - 1) / (kFinWarps * gx) + kFinSetup);
        if (cost < least) {
          least = cost;
          best  = gx;
        }
      }
      return best;
    }

    template <int C>
    int launch_finish(const MomentFinishParams& r, dim3 grid, size_t smem, cudaStream_t s) {
      static std::atomic<uint64_t> configured { 0 };
      RG_CUDA_TRY(ensure_max_dynamic_smem(moments_finish_kernel<C>,
                                          static_cast<int>(finish_smem(32 * C - 1, kMomMaxTable)), configured));
      moments_finish_kernel<C><<<grid, kFinThreads, smem, s>>>(r);
      RG_CUDA_TRY(cudaGetLastError());
      return RG_OK;
    }

  } // namespace

  // The row sums and every bin's sum over its cells, into out (nseg x nbins).
  int moments_finish(rg_spectrum_plan* pl, int nseg, float* out, cudaStream_t s) {
    if (pl->aligned) {
      return smooth_moments_finish(pl, nseg, out, s);
    }
    DeviceContext* ctx = nullptr;
    RG_TRY(context(&ctx));
    MomentFinishParams r {};
    r.hist     = pl->d_hist;
    r.per_seg  = pl->hist_per_seg;
    r.mslice   = reinterpret_cast<const int4*>(pl->d_mslice);
    r.bins     = pl->d_binfo;
    r.coef     = pl->d_mcoef;
    r.nseg_tab = pl->ref->n - 1;
    r.nslices  = pl->nslices;
    r.nbins    = pl->nbins;
    r.ebins    = pl->d_ebins;
    r.status   = pl->d_status;
    r.acc      = pl->d_msum;
    r.done     = reinterpret_cast<unsigned*>(pl->d_msum + pl->msum_cap * kSliceBins);
    r.out      = out;
    r.nz       = negative_zeros();
    const int    rows   = nseg * pl->nslices;
    const int    nv     = max_valid(pl);
    const size_t smem   = finish_smem(nv, r.nseg_tab);
    const int    gx     = finish_blocks(rows, max_cells(pl), ctx->sms * std::max(1, static_cast<int>(kFinSmSmem / (smem + 1024))));
    const dim3   grid(gx, rows);
    int          st = RG_OK;
    switch ((nv + 1 + 31) / 32) {
#define RG_C_CASE(c)                                                                         \
  case c:                                                                                    \
    st = launch_finish<c>(r, grid, smem, s);                                                 \
    break;
      RG_C_CASE(1) RG_C_CASE(2) RG_C_CASE(3) RG_C_CASE(4) RG_C_CASE(5) RG_C_CASE(6) RG_C_CASE(7) RG_C_CASE(8)
      RG_C_CASE(9) RG_C_CASE(10) RG_C_CASE(11) RG_C_CASE(12) RG_C_CASE(13) RG_C_CASE(14) RG_C_CASE(15)
      RG_C_CASE(16) RG_C_CASE(17)
#undef RG_C_CASE
      default:
        return set_error(RG_ERR_UNSUPPORTED, "more than 512 bins in a slice");
    }
    RG_TRY(st);
    pl->hist_dirty = pl->hist_stays_dirty;
    return RG_OK;
  }

  void moments_free(rg_spectrum_plan* pl) {
    cudaFree(pl->d_mslice);
    cudaFree(pl->d_mrange);
    cudaFree(pl->d_thr);
    cudaFree(pl->d_bucket);
    cudaFree(pl->d_binfo);
    cudaFree(pl->d_mcoef);
    cudaFree(pl->d_hist);
    cudaFree(pl->d_msum);
    cudaFree(pl->d_logt);
    cudaFree(pl->d_cells);
    cudaFree(pl->own_smooth.d_coef);
    pl->d_cells           = nullptr;
    pl->cells_cap         = 0;
    pl->own_smooth.d_coef = nullptr;
    pl->d_mslice = nullptr;
    pl->d_mrange = nullptr;
    pl->d_thr    = nullptr;
    pl->d_bucket = nullptr;
    pl->d_binfo  = nullptr;
    pl->d_mcoef  = nullptr;
    pl->d_hist   = nullptr;
    pl->hist_cap = 0;
    pl->d_msum   = nullptr;
    pl->msum_cap = 0;
    pl->d_logt   = nullptr;
  }

} // namespace rg

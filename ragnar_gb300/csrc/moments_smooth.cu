// Differentiable (smooth-table) particle spectrum and its adjoint by cell moments.
//
// Reference path: SynchrotronSpectrum<D> (synchrotron.cpp:107-145) over
// sync::Kernel<D>::operator() (synchrotron.hpp:145-172); the smooth table is this
// library's own differentiable F (exact x int K_{5/3} at the nodes, C1 cubic
// Hermite in between; ftable.cu).
//
// For photon bins that are log-uniform (Logbins), a plan builds its own smooth
// table on a grid aligned to the bins: node spacing dln = (bin spacing) / m for an
// integer m, and nodes placed so that every bin's table coordinate t_b is an
// integer up to a tiny residual eps_b (float rounding of the bins; |eps_b| < 1e-3
// segments).  With x = e_b / e_peak, t = t_b - q_p, q_p = ln e_peak_p / dln, every
// bin then sees a particle at the same position inside a segment,
//   tau_p = frac(-q_p),   segment s = t_b - ceil(q_p),
// so with R = Pmax - Q (Q = q 2^F in fixed point, Pmax the largest bin coordinate)
// a particle's cell Rc = R >> F and tau = (R mod 2^F) 2^-F are the same for every
// bin, and bin b reads segment Rc - Dc_b (Dc_b = (Pmax >> F) - t_b).  The forward is
//   S_b / e_b = sum_cells sum_j c'_j(Rc - Dc_b) M_j(Rc),  M_j = sum_p A_p tau_p^j,
//   c'_j = c_j + eps_b (j + 1) c_{j+1}   (first order in eps_b: F(tau + eps)),
// four FP64 moments per cell (deposited into kSub slots per cell, which spreads the
// atomics of crowded cells), and the adjoint of a loss L with
// G_b = dL/dS_b is, per particle, the cubic of its cell
//   R1(tau) = sum_b G_b e_b F_b(tau) = sum_j alpha_j(Rc) tau^j,
//   alpha_j(c) = sum_b G_b e_b c'_j(c - Dc_b),   R2 = (dR1/dtau) / dln,
// from which particle_gradient forms dL/dw and dL/du.  Work: one particle stage per
// particle plus (cells x bins) in the forward and the adjoint, instead of
// (particles x bins) in each.
#include "pair_stage.cuh"

#include <algorithm>
#include <cmath>
#include <cstring>
#include <limits>
#include <type_traits>
#include <vector>

namespace rg {

  namespace {

    // Slots per cell: a particle adds its moments (which are absolute within the cell) to
    // the slot of its lane, shifted by its position in the cell, so the lanes of a warp
    // whose particles crowd one cell hit different addresses.
    constexpr int    kSub         = 32;
    constexpr int    kSubBits     = 5;
    constexpr int    kSmBlocksPerSM = 2;
    constexpr int    kSmAdjBlocksPerSM = 3;
    constexpr double kTargetDln   = 0.0089954; // ln(1e8) / 2048: the device-wide table's spacing
    // Largest bin residual |eps_b|, in table segments.  Logbins-style bins carry ~2e-6 in
    // ln e (their exponent is rounded to float before the power); the first-order
    // correction leaves eps^2 |F''| / 2 < 1e-6 F at this bound.
    constexpr double kUniformTol  = 1e-3;

    struct SmoothMomParams {
      FusedParams    fp;        // kinematics constants (plan's frac), status
      LogParams      log;
      PairStreams    in;
      int64_t        Pmin, Pmax, L;
      int            F;         // fraction bits of the coordinate (plan frac + 8)
      float          tau_scale; // 2^-F
      int            nc;        // cells
      double*        hist;      // [nseg][nc][kSub][4]
      RunSums        run;       // the deposit's
      uint2*         place;     // single-segment runs: per particle (cell, fraction bits) or
                                // (kNoCell, 0) for a particle that adds nothing; null: not kept
    };

    constexpr uint32_t kNoCell = 0xffffffffu;

    // A pair's cells and fraction bits; kNoCell for a particle that adds nothing (a zero weight
    // still has a cell: its gradient is not zero).
    __device__ __forceinline__ void cells_of(const Place2& pl, const SmoothMomParams& m, uint32_t (&cell)[2],
                                             uint32_t (&Rl)[2]) {
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const int64_t c = pl.Y[j] >> (m.F + m.log.fx);
        Rl[j]           = static_cast<uint32_t>(pl.Y[j] >> m.log.fx) & ((1u << m.F) - 1u);
        cell[j]         = static_cast<uint64_t>(c) < static_cast<uint64_t>(m.nc) && fabsf(pl.A[j]) <= 3.402823466e38f
                            ? static_cast<uint32_t>(c)
                            : kNoCell;
      }
    }

    // The four moments of every lane's particle into its entry (idx, in units of four doubles;
    // kNoEntry for none).  The L2 takes one request per 32-byte sector and instruction, so the
    // four lanes of a quad add one particle's four moments in one instruction, then the next
    // lane's: 1.27e11 particles/s on random entries of a 4 MB table, against 5.1e10 when each
    // lane adds its own four in turn.  Called by whole warps.
    __device__ __forceinline__ void red_quad(double* hist, uint32_t idx, float A, float tau) {
      const int  lane = threadIdx.x & 31;
      const bool o1 = lane & 1, o2 = lane & 2;
      // 4 x 4 transpose within the quad: t[k] = this lane's moment of lane k's particle
      const float a1 = A * tau, a2 = a1 * tau, a3 = a2 * tau;
      const float x0 = __shfl_xor_sync(0xffffffffu, o1 ? A : a1, 1), x1 = __shfl_xor_sync(0xffffffffu, o1 ? a2 : a3, 1);
      const float p0 = o1 ? x0 : A, p1 = o1 ? a1 : x0; // moment (lane & 1) of the pair's even, odd particle
      const float q0 = o1 ? x1 : a2, q1 = o1 ? a3 : x1; // moment 2 + (lane & 1)
      const float y0 = __shfl_xor_sync(0xffffffffu, o2 ? p0 : q0, 2), y1 = __shfl_xor_sync(0xffffffffu, o2 ? p1 : q1, 2);
      const float t[4] = { o2 ? y0 : p0, o2 ? y1 : p1, o2 ? q0 : y0, o2 ? q1 : y1 };
      double*     mine = hist + (lane & 3);
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const uint32_t i = __shfl_sync(0xffffffffu, idx, (lane & ~3) | k);
        red_add_if(i != kNoEntry, mine + 4 * static_cast<size_t>(i), static_cast<double>(t[k]));
      }
    }

    // Two particles per thread and step, as the interval-moment deposit (moments.cu).  Measured on
    // 1e7 particles (|u| ~ u^-2, B along z) x 512 bins: 120 us (8.4e10 particles/s) against 229 us
    // for one particle per thread with four requests of its own; the L2's reduction requests set
    // its pace (32 slots time as 64, three blocks per SM as two; the floats turned into doubles by
    // integer instructions instead of the FP64 pipe 124 us).
    template <bool kE, bool kSeg>
    __global__ void __launch_bounds__(kPairThreads, kSmBlocksPerSM)
      smooth_deposit_kernel(const __grid_constant__ SmoothMomParams m) {
      __shared__ int64_t  logt[kLogEntries];
      __shared__ uint32_t soff[kSeg ? kPairSharedSeg + 1 : 1];
      clear_run_sums(m.run);
      stage_log_table(m.log, m.log.fx, m.Pmax, logt, kPairThreads);
      if (!stage_segments<kSeg>(m.in, m.fp.status, soff)) {
        return;
      }
      const uint32_t first = kSeg ? soff[0] : 0u;
      const uint32_t last  = kSeg ? soff[m.in.nseg] : static_cast<uint32_t>(min(m.in.n - m.in.window, kPairWindow));
      const uint32_t step  = gridDim.x * kPairChunk, tid = threadIdx.x;
      uint32_t       useg = 0, uend = kSeg ? soff[1] : last; // the segment of the step's first particle, and its end
      auto           add  = [&](uint32_t base, const float2 (&from)[kComps]) {
        f2 v[kComps];
        to_pairs<kE>(from, v);
        const Place2 pl = place2<kE>(v, m.fp, m.log, logt, m.Pmin, m.Pmax, m.L);
        if (kSeg) {
          while (uend <= base) { // base < last = soff[nseg]
            ++useg;
            uend = soff[useg + 1];
          }
        }
        uint32_t cell[2], Rl[2], idx[2];
        cells_of(pl, m, cell, Rl);
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const uint32_t i   = base + tid + j * kPairThreads;
          const uint32_t sub = ((Rl[j] >> (m.F - kSubBits)) + tid) & (kSub - 1);
          bool           on  = cell[j] != kNoCell && i < last;
          uint32_t       seg = useg;
          if (kSeg && on) {
            while (soff[seg + 1] <= i) { // i < soff[nseg]
              ++seg;
            }
          }
          idx[j] = on ? (seg * static_cast<uint32_t>(m.nc) + cell[j]) * kSub + sub : kNoEntry;
          if (!kSeg && m.place && i < last) {
            m.place[i] = make_uint2(cell[j], cell[j] == kNoCell ? 0u : Rl[j]);
          }
        }
        __syncwarp();
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          red_quad(m.hist, idx[j], pl.A[j], __uint2float_rn(Rl[j]) * m.tau_scale);
        }
      };
      constexpr int kSets = kE ? 2 : 3;
      float2        set[kSets][kComps];
      uint32_t      base = first + blockIdx.x * kPairChunk;
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

    // ---- finish: cells folded, then every bin over the block's cells ---------------------------
    struct SmoothFinishParams {
      double*         hist;  // read, and set back to zero for the next run
      int             nc;
      const int4*     binfo; // per bin: (Dc, eps bits, 0, valid)
      const float4*   coef;
      int             nseg_tab;
      int             nbins;
      const float*    ebins;
      const unsigned* status;
      double*         acc;   // [nseg][acc_stride], cleared by the deposit
      unsigned*       done;  // [nseg] blocks finished, cleared by the deposit
      int             acc_stride;
      float*          out;   // nseg x nbins
      f2              nz;    // of product2
    };

    constexpr int kFinCells = 16; // cells per block: two per warp
    // Cells up to 2^-kFinBelow of the block's largest keep all their bits in its packed sums, whose products
    // with coefficients down to the smallest float (the table's far end) are kept exact by the
    // moments' unit 2^-kFinUnit; blocks whose cells span more (a particle that outweighs others by
    // 1e18) sum in FP64.
    constexpr int kFinBelow = 60, kFinUnit = 60;

    // Block: kFinCells cells of one segment (blockIdx.y).  Its warps sum the cells' slots in FP64 and
    // clear them, and leave the cells that hold anything in shared memory as double-floats scaled
    // by a power of two; then every thread takes bins,
    //   S_b / e_b += sum_cells sum_j c'_j(c - Dc_b) M_j(c),  c'_j = c_j + eps_b (j + 1) c_{j+1},
    // two cells at a time in packed double-floats (2^-44; the FP64 pipe issues 1.6 operations per
    // clock and SM: a fold kernel and an FP64 reduction per bin took 9 + 22 us for 512 bins x 4826
    // cells, this kernel 15 us).  eps_b B, B = sum (j + 1) c_{j+1} M_j, is summed in FP32:
    // |eps_b| < 1e-3, so its rounding is below 1e-10 of the sum.  The blocks add their bins in FP64
    // and the last block of a segment writes the spectrum.
    __global__ void __launch_bounds__(kPairThreads) smooth_finish_kernel(const __grid_constant__ SmoothFinishParams r) {
      extern __shared__ float4 coef[]; // nseg_tab
      __shared__ double sums[kFinCells][4];
      __shared__ float4 Mh[kFinCells + 1], Ml[kFinCells + 1]; // moments of the block's live cells, hi and lo
      __shared__ int    live[kFinCells + 1], nlive, scale;
      __shared__ bool   wide, last;
      const int  seg = blockIdx.y, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
      const int  c0 = blockIdx.x * kFinCells, ncell = min(kFinCells, r.nc - c0);
      const bool failed = *r.status != kDevOk;
      // A warp takes two cells, all loads issued first; lane l holds moments (0, 1) or (2, 3) (l even
      // or odd) of slots l / 2 and l / 2 + 16, and the slots are summed by halving: each exchange
      // leaves a lane half of its values (a shuffle sum of each would be four times the FP64 adds).
      static_assert(kSub == 32 && kFinCells == 2 * (kPairThreads / 32), "two cells of 32 slots per warp");
      const int cell0 = 2 * warp;
      double2*  h     = reinterpret_cast<double2*>(r.hist + (static_cast<int64_t>(seg) * r.nc + c0 + cell0) * kSub * 4) + lane;
      double2   d[2][2];
#pragma unroll
      for (int k = 0; k < 2; ++k) {
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          d[k][q] = cell0 + k < ncell ? h[k * kSub * 2 + 32 * q] : make_double2(0.0, 0.0);
        }
      }
      for (int i = threadIdx.x; i < r.nseg_tab; i += kPairThreads) {
        coef[i] = __ldg(r.coef + i);
      }
      bool any = false;
#pragma unroll
      for (int k = 0; k < 2; ++k) {
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          any = any || d[k][q].x != 0.0 || d[k][q].y != 0.0;
        }
      }
      double t = 0.0;
      if (__any_sync(0xffffffffu, any)) {
#pragma unroll
        for (int k = 0; k < 2; ++k) {
#pragma unroll
          for (int q = 0; q < 2; ++q) {
            if (cell0 + k < ncell) {
              h[k * kSub * 2 + 32 * q] = make_double2(0.0, 0.0);
            }
          }
        }
        const bool b4 = lane & 16, b3 = lane & 8;
        const double x0 = d[0][0].x + d[0][1].x, y0 = d[0][0].y + d[0][1].y;
        const double x1 = d[1][0].x + d[1][1].x, y1 = d[1][0].y + d[1][1].y;
        const double x = (b4 ? x1 : x0) + __shfl_xor_sync(0xffffffffu, b4 ? x0 : x1, 16); // cell: bit 4
        const double y = (b4 ? y1 : y0) + __shfl_xor_sync(0xffffffffu, b4 ? y0 : y1, 16);
        t = (b3 ? y : x) + __shfl_xor_sync(0xffffffffu, b3 ? x : y, 8);                     // moment: bits 0 and 3
        t += __shfl_xor_sync(0xffffffffu, t, 4);
        t += __shfl_xor_sync(0xffffffffu, t, 2);
      }
      if ((lane & 6) == 0) {
        sums[cell0 + (lane >> 4)][2 * (lane & 1) + ((lane >> 3) & 1)] = t;
      }
      __syncthreads();
      if (warp == 0) { // the live cells in order, and the scale: the largest exponent
        int top = 0, low = 0x7ff; // the cell's largest exponent; that of its sum of amplitudes
        if (lane < ncell) {
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            top = max(top, (__double2hiint(sums[lane][j]) >> 20) & 0x7ff);
          }
          low = top > 0 ? (__double2hiint(sums[lane][0]) >> 20) & 0x7ff : 0x7ff;
        }
        low = __reduce_min_sync(0xffffffffu, low);
        const unsigned on  = __ballot_sync(0xffffffffu, top > 0);
        const int      all = __reduce_max_sync(0xffffffffu, top) - 1023;
        if (top > 0) {
          const int at = __popc(on & ((1u << lane) - 1u));
          float2    f[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            f[j] = split_double(sums[lane][j], all - kFinUnit);
          }
          live[at] = c0 + lane;
          Mh[at]   = make_float4(f[0].x, f[1].x, f[2].x, f[3].x);
          Ml[at]   = make_float4(f[0].y, f[1].y, f[2].y, f[3].y);
        }
        if (lane == 0) {
          const int n = __popc(on);
          live[n]     = -1; // the second cell of an odd last pair: in no bin's table
          Mh[n] = Ml[n] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
          nlive = n;
          scale = all - kFinUnit;
          wide  = all + 1023 - low > kFinBelow;
        }
      }
      __syncthreads();
      const int n     = nlive;
      double*   total = r.acc + static_cast<int64_t>(seg) * r.acc_stride;
      if (n > 0 && !failed && wide) {
        for (int b = threadIdx.x; b < r.nbins; b += kPairThreads) {
          const int4 bi = r.binfo[b];
          double     A = 0.0, B = 0.0;
          for (int k = 0; k < n && bi.w; ++k) {
            const int s = live[k] - bi.x;
            if (s >= 0 && s < r.nseg_tab) {
              const double* M = sums[live[k] - c0];
              const float4  c = coef[s];
              A += c.x * M[0] + c.y * M[1] + c.z * M[2] + c.w * M[3];
              B += c.y * M[0] + 2.0 * c.z * M[1] + 3.0 * c.w * M[2];
            }
          }
          const double t = A + static_cast<double>(__int_as_float(bi.y)) * B;
          if (t != 0.0) {
            atomicAdd(total + b, t);
          }
        }
      } else if (n > 0 && !failed) {
        const double s2 = __hiloint2double((scale + 1023) << 20, 0);
        for (int b = threadIdx.x; b < r.nbins; b += kPairThreads) {
          const int4 bi = r.binfo[b];
          if (!bi.w || live[n - 1] < bi.x || live[0] >= bi.x + r.nseg_tab) {
            continue;
          }
          ff2 A { set2(0.0f), set2(0.0f) };
          f2  B = set2(0.0f);
          for (int k = 0; k < n; k += 2) {
            const int    sa = live[k] - bi.x, sb = live[k + 1] - bi.x;
            const bool   oa = sa >= 0 && sa < r.nseg_tab, ob = sb >= 0 && sb < r.nseg_tab;
            const float4 z = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            const float4 ca = oa ? coef[sa] : z, cb = ob ? coef[sb] : z;
            const float4 ha = Mh[k], hb = Mh[k + 1], la = Ml[k], lb = Ml[k + 1];
            const f2     c[4] = { pack2(ca.x, cb.x), pack2(ca.y, cb.y), pack2(ca.z, cb.z), pack2(ca.w, cb.w) };
            const f2     h[4] = { pack2(ha.x, hb.x), pack2(ha.y, hb.y), pack2(ha.z, hb.z), pack2(ha.w, hb.w) };
            const f2     l[4] = { pack2(la.x, lb.x), pack2(la.y, lb.y), pack2(la.z, lb.z), pack2(la.w, lb.w) };
            // c_j (h_j + l_j): the products, summed pairwise, and what lies below them
            f2 p[4], e[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              p[j] = product2(c[j], h[j], r.nz);
              e[j] = sub2(mul2(c[j], l[j]), fma2(neg2(c[j]), h[j], p[j]));
            }
            const ff2 s01 = two_sum2(p[0], p[1]), s23 = two_sum2(p[2], p[3]);
            const ff2 s4  = two_sum2(s01.hi, s23.hi), t = two_sum2(A.hi, s4.hi);
            const f2  low = add2(add2(add2(e[0], e[1]), add2(e[2], e[3])), add2(add2(s01.lo, s23.lo), s4.lo));
            A             = fast_two_sum2(t.hi, add2(t.lo, add2(A.lo, low)));
            B = add2(B, fma2(c[1], h[0], fma2(mul2(c[2], set2(2.0f)), h[1], mul2(mul2(c[3], set2(3.0f)), h[2]))));
          }
          float h0, h1, l0, l1, b0, b1;
          unpack2(A.hi, h0, h1);
          unpack2(A.lo, l0, l1);
          unpack2(B, b0, b1);
          const ff     a = ff_add(ff_add(ff { h0, l0 }, ff { h1, l1 }), two_prod(__int_as_float(bi.y), b0 + b1));
          const double t = (static_cast<double>(a.hi) + static_cast<double>(a.lo)) * s2;
          if (t != 0.0) {
            atomicAdd(total + b, t);
          }
        }
      }
      __threadfence();
      __syncthreads();
      if (threadIdx.x == 0) {
        last = atomicAdd(r.done + seg, 1u) == gridDim.x - 1;
      }
      __syncthreads();
      if (!last) {
        return;
      }
      __threadfence();
      for (int b = threadIdx.x; b < r.nbins; b += kPairThreads) {
        const double t = __ldcg(total + b);
        r.out[static_cast<int64_t>(seg) * r.nbins + b] =
          failed ? __int_as_float(0x7fffffff) : __double2float_rn(t * static_cast<double>(r.ebins[b]));
      }
    }

    // alpha_j(c) = sum_b G_b e_b c'_j(c - Dc_b) for every cell of a segment (blockIdx.y): one warp per
    // cell, its lanes taking every 32nd bin with FP32 products and compensated (Kahan) sums, two
    // coefficients per packed instruction, then a double-float sum over the lanes in a fixed
    // order.  The bins' (G_b e_b, eps_b, Dc_b) are staged once per block (9.3 us for 512 bins x 4826
    // cells, 11.7 us without the staging and with scalar sums).
    struct SmoothAlphaParams {
      const float*  grad_out; // nseg x nbins
      const int4*   binfo;
      const float4* coef;
      int           nseg_tab;
      int           nbins;
      const float*  ebins;
      int           nc;
      float4*       alpha; // nseg x nc
    };

    __device__ __forceinline__ void kahan_add2(f2& s, f2& c, f2 x) {
      const f2 y = sub2(x, c);
      const f2 t = add2(s, y);
      c          = sub2(sub2(t, s), y);
      s          = t;
    }

    constexpr int kSmAlphaThreads = 256;
    constexpr int kSmAlphaBins    = 1024; // bins staged at a time

    __global__ void __launch_bounds__(kSmAlphaThreads) smooth_alpha_kernel(const __grid_constant__ SmoothAlphaParams a) {
      __shared__ float3 bins[kSmAlphaBins]; // G_b e_b (0 for a bin that is not valid), eps_b, Dc_b (bits)
      const int seg = blockIdx.y, lane = threadIdx.x & 31;
      const int c = blockIdx.x * (kSmAlphaThreads / 32) + (threadIdx.x >> 5);
      f2        s01 = set2(0.0f), s23 = set2(0.0f), e01 = set2(0.0f), e23 = set2(0.0f);
      for (int b0 = 0; b0 < a.nbins; b0 += kSmAlphaBins) {
        const int m = min(kSmAlphaBins, a.nbins - b0);
        __syncthreads();
        for (int i = threadIdx.x; i < m; i += kSmAlphaThreads) {
          const int4 bi = __ldg(a.binfo + b0 + i);
          bins[i]       = make_float3(__ldg(a.grad_out + static_cast<int64_t>(seg) * a.nbins + b0 + i) * __ldg(a.ebins + b0 + i),
                                      __int_as_float(bi.y), __int_as_float(bi.w ? bi.x : 0x7fffffff));
        }
        __syncthreads();
        if (c < a.nc) {
#pragma unroll 4
          for (int i = lane; i < m; i += 32) {
            const float3 b  = bins[i];
            const int    sg = c - __float_as_int(b.z); // negative for a bin that is not valid
            if (sg >= 0 && sg < a.nseg_tab) {
              const float4 k = __ldg(a.coef + sg);
              kahan_add2(s01, e01, pack2(b.x * fmaf(b.y, k.y, k.x), b.x * fmaf(2.0f * b.y, k.z, k.y)));
              kahan_add2(s23, e23, pack2(b.x * fmaf(3.0f * b.y, k.w, k.z), b.x * k.w));
            }
          }
        }
      }
      if (c >= a.nc) {
        return;
      }
      float s[4], e[4];
      unpack2(s01, s[0], s[1]);
      unpack2(s23, s[2], s[3]);
      unpack2(e01, e[0], e[1]);
      unpack2(e23, e[2], e[3]);
      float out[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        // the lane's sum is s - e; add the lanes' double-floats pairwise
        ff v = fast_two_sum(s[j], -e[j]);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
          const float oh = __shfl_xor_sync(0xffffffffu, v.hi, o);
          const float ol = __shfl_xor_sync(0xffffffffu, v.lo, o);
          // every lane forms the same sum in the same order: the lower lane's value first
          const bool lower = (lane & o) == 0;
          const ff   x = lower ? v : ff { oh, ol }, y = lower ? ff { oh, ol } : v;
          const ff   h = two_sum(x.hi, y.hi);
          v            = fast_two_sum(h.hi, __fadd_rn(h.lo, __fadd_rn(x.lo, y.lo)));
        }
        out[j] = __fadd_rn(v.hi, v.lo);
      }
      if (lane == 0) {
        a.alpha[static_cast<int64_t>(seg) * a.nc + c] = make_float4(out[0], out[1], out[2], out[3]);
      }
    }

    struct SmoothAdjParams {
      SmoothMomParams m;
      const uint2*    place; // a forward's placement record (single segment), or null: recompute
      const float4*   alpha; // nseg x nc
      float           inv_dln;
      float*          gw;
      float*          gu[3];
    };

    // dL/dw and dL/du of two particles without an E field, as particle_gradient (same formulas,
    // the cross product in double-floats); bit j of the result: particle j is done, otherwise it
    // takes the scalar form (ranges in which the reciprocals below would leave FP32's normal numbers).
    __device__ __forceinline__ unsigned gradient2(const f2 (&v)[kComps], float amp, f2 R1, f2 R2, f2& gw, f2 (&gu)[3], f2 nz) {
      const f2  u[3] = { v[0], v[1], v[2] }, B[3] = { v[6], v[7], v[8] };
      const f2  n[3] = { neg2(u[0]), neg2(u[1]), neg2(u[2]) };
      const f2  G    = fma2(u[0], u[0], fma2(u[1], u[1], fma2(u[2], u[2], set2(1.0f))));
      const f2  c[3] = { diff_of_products2(u[1], n[1], B[2], u[2], n[2], B[1], nz).hi,
                         diff_of_products2(u[2], n[2], B[0], u[0], n[0], B[2], nz).hi,
                         diff_of_products2(u[0], n[0], B[1], u[1], n[1], B[0], nz).hi };
      const f2  W    = fma2(c[2], c[2], fma2(c[1], c[1], mul2(c[0], c[0])));
      const f2  nc[3] = { neg2(c[0]), neg2(c[1]), neg2(c[2]) };
      // d W / du / 2 = B x c
      const f2  x[3] = { fma2(B[1], c[2], mul2(B[2], nc[1])), fma2(B[2], c[0], mul2(B[0], nc[2])),
                         fma2(B[0], c[1], mul2(B[1], nc[0])) };
      float g[2], w[2], rg[2], rw[2], y[2];
      unpack2(G, g[0], g[1]);
      unpack2(W, w[0], w[1]);
      unsigned ok = 0;
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        ok |= (g[j] <= 1e15f && w[j] >= 1e-20f && w[j] <= 1e30f ? 1u : 0u) << j; // not for NaN
        rg[j] = rcp_approx(g[j]);
        rw[j] = rcp_approx(w[j]);
      }
      // 1/G and 1/W with one correction each, W / G, and its square root with one
      const f2 one = set2(1.0f), G1 = pack2(rg[0], rg[1]), W1 = pack2(rw[0], rw[1]);
      const f2 iG = fma2(G1, fma2(neg2(G), G1, one), G1), iW = fma2(W1, fma2(neg2(W), W1, one), W1);
      const f2 q0 = mul2(W, iG);
      const f2 q  = fma2(fma2(neg2(q0), G, W), iG, q0);
      float    qq[2];
      unpack2(q, qq[0], qq[1]);
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y[j]) : "f"(qq[j]));
      }
      const f2 yy = pack2(y[0], y[1]), s0 = mul2(q, yy);
      const f2 chi = mul2(fma2(fma2(neg2(s0), s0, q), mul2(yy, set2(0.5f)), s0), set2(amp));
      const f2 A   = mul2(chi, v[9]);
      const f2 nR2 = neg2(R2);
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        const f2 b   = mul2(u[d], iG);
        const f2 chd = fma2(x[d], iW, neg2(b)), epd = fma2(x[d], iW, b); // d ln chiR, d ln e_peak
        gu[d]        = mul2(A, fma2(R1, chd, mul2(nR2, epd)));
      }
      gw = mul2(chi, R1);
      return ok;
    }

    // Per pair: the cells (from the record, or placed again as the forward did), the cells' cubics,
    // and the chain rule.  28 B read and 16 B written per particle, and 8 B of record.  Measured on
    // the deposit's 1e7 particles: 78 us (6.6 TB/s, 0.98 of the measured copy) with the record,
    // against 99 us with the scalar gradient (268 instructions a particle, now 148).
    template <bool kE, bool kSeg, bool kPlaced>
    __global__ void __launch_bounds__(kPairThreads, kSmAdjBlocksPerSM)
      smooth_adjoint_kernel(const __grid_constant__ SmoothAdjParams a) {
      __shared__ int64_t     logt[kPlaced ? 1 : kLogEntries];
      __shared__ uint32_t    soff[kSeg ? kPairSharedSeg + 1 : 1];
      const SmoothMomParams& m = a.m;
      if (!kPlaced) {
        stage_log_table(m.log, m.log.fx, m.Pmax, logt, kPairThreads);
      }
      if (!stage_segments<kSeg>(m.in, m.fp.status, soff)) {
        return;
      }
      const uint32_t first = kSeg ? soff[0] : 0u;
      const uint32_t last  = kSeg ? soff[m.in.nseg] : static_cast<uint32_t>(min(m.in.n - m.in.window, kPairWindow));
      const uint32_t step  = gridDim.x * kPairChunk, tid = threadIdx.x;
      uint32_t       useg = 0, uend = kSeg ? soff[1] : last;
      uint2          rec[2], rec_next[2];
      auto           load_record = [&](uint32_t base) {
        if (kPlaced) {
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            const uint32_t i = base + tid + j * kPairThreads;
            rec_next[j]      = i < last ? __ldg(a.place + i) : make_uint2(kNoCell, 0u);
          }
        }
      };
      float2   next[kComps];
      uint32_t base = first + blockIdx.x * kPairChunk;
      load_pair<kE>(m.in, base, last, next);
      load_record(base);
      for (; base < last; base += step) {
        f2 v[kComps];
        to_pairs<kE>(next, v);
        rec[0] = rec_next[0];
        rec[1] = rec_next[1];
        load_pair<kE>(m.in, base + step, last, next);
        load_record(base + step);
        uint32_t cell[2], Rl[2];
        if (kPlaced) {
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            cell[j] = rec[j].x;
            Rl[j]   = rec[j].y;
            if (cell[j] != kNoCell && cell[j] >= static_cast<uint32_t>(m.nc)) { // a record of another plan
              atomicOr(m.fp.status, kDevBadIndex);
              cell[j] = kNoCell;
            }
          }
        } else {
          const Place2 pl = place2<kE>(v, m.fp, m.log, logt, m.Pmin, m.Pmax, m.L);
          cells_of(pl, m, cell, Rl);
        }
        if (kSeg) {
          while (uend <= base) { // base < last = soff[nseg]
            ++useg;
            uend = soff[useg + 1];
          }
        }
        float R1[2], R2[2];
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const uint32_t i   = base + tid + j * kPairThreads;
          uint32_t       seg = useg;
          if (kSeg && i < last) {
            while (soff[seg + 1] <= i) { // i < soff[nseg]
              ++seg;
            }
          }
          const float  tau = __uint2float_rn(Rl[j]) * m.tau_scale;
          const float4 al  = cell[j] != kNoCell && i < last
                               ? __ldg(a.alpha + static_cast<int64_t>(seg) * m.nc + cell[j])
                               : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
          R1[j] = fmaf(tau, fmaf(tau, fmaf(tau, al.w, al.z), al.y), al.x);
          R2[j] = fmaf(tau, fmaf(tau, 3.0f * al.w, 2.0f * al.z), al.y) * a.inv_dln;
        }
        float    gw[2], gu[3][2];
        unsigned done = 0;
        if (!kE) {
          f2 gw2, gu2[3];
          done = gradient2(v, m.fp.amp, pack2(R1[0], R1[1]), pack2(R2[0], R2[1]), gw2, gu2, m.log.nz);
          unpack2(gw2, gw[0], gw[1]);
#pragma unroll
          for (int d = 0; d < 3; ++d) {
            unpack2(gu2[d], gu[d][0], gu[d][1]);
          }
        }
        if (done != 3u) {
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            if (!((done >> j) & 1u)) {
              float s[kComps], g1, g3[3];
#pragma unroll
              for (int c = 0; c < kComps; ++c) {
                float lo, hi;
                unpack2(v[c], lo, hi);
                s[c] = j ? hi : lo;
              }
              particle_gradient(s, m.fp, R1[j], R2[j], g1, g3);
              gw[j] = g1;
#pragma unroll
              for (int d = 0; d < 3; ++d) {
                gu[d][j] = g3[d];
              }
            }
          }
        }
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const uint32_t i    = base + tid + j * kPairThreads;
          const bool     live = cell[j] != kNoCell; // others have no gradient
          if (i < last) {
            if (a.gw) {
              a.gw[i] = live ? gw[j] : 0.0f;
            }
#pragma unroll
            for (int d = 0; d < 3; ++d) {
              if (a.gu[d]) {
                a.gu[d][i] = live ? gu[d][j] : 0.0f;
              }
            }
          }
        }
      }
    }

    void fill_smooth_params(rg_spectrum_plan* pl, const float* const comp[kComps], const int64_t* d_off, int64_t n,
                            int nseg, SmoothMomParams& m) {
      m = SmoothMomParams {};
      fill_params(pl, comp, nullptr, nullptr, n, 1, m.fp);
      fill_log_params(pl, m.log);
      m.Pmin      = pl->sm_pmin;
      m.Pmax      = pl->sm_pmax;
      m.L         = pl->mom_L;
      m.F         = pl->frac + 8;
      m.tau_scale = std::ldexp(1.0f, -m.F);
      m.nc        = pl->sm_cells;
      m.hist      = reinterpret_cast<double*>(pl->d_hist);
    }

  } // namespace

  // A plan's own smooth table aligned to log-uniform bins (see the file comment); leaves
  // the plan on the device-wide table when the bins are not log-uniform or the table
  // would need more than kSmoothMaxSegments segments.  ln_k0 = ln(eps / (g^2 B0)).
  int smooth_align_plan(rg_spectrum_plan* pl, double ln_k0) {
    const int n = pl->nbins;
    if (n < 2) {
      return RG_OK;
    }
    std::vector<double> le(n);
    for (int b = 0; b < n; ++b) {
      const double e = pl->h_bins[b];
      if (!(e > 0.0) || !std::isfinite(e)) {
        return RG_OK;
      }
      le[b] = std::log(e);
    }
    const double step = (le[n - 1] - le[0]) / (n - 1);
    if (!(step > 0.0)) {
      return RG_OK;
    }
    const int    m   = static_cast<int>(std::ceil(step / kTargetDln));
    const double dln = step / m;
    for (int b = 0; b < n; ++b) {
      if (std::fabs(le[b] - le[0] - b * step) > kUniformTol * dln) {
        return RG_OK;
      }
    }
    // nodes at ln e_0 - ln K0 - k dln, with the first node at or below x = 1e-6 and the
    // last at or above x = 100 (the device-wide table's range)
    const double base  = le[0] - ln_k0;
    const double k     = std::ceil((base - std::log(kSmoothXmin)) / dln);
    const double ln_x0 = base - k * dln;
    const double nseg  = std::ceil((std::log(kSmoothXmax) - ln_x0) / dln);
    if (!(nseg >= 1.0) || nseg > kSmoothMaxSegments) {
      return RG_OK;
    }
    RG_TRY(build_smooth_table_geom(pl->own_smooth, ln_x0, dln, static_cast<int>(nseg), nullptr));
    pl->smooth  = &pl->own_smooth;
    pl->aligned = true;
    return RG_OK;
  }

  // Cell tables of an aligned smooth plan (after its bins' fixed-point preparation).
  int smooth_moments_prepare(rg_spectrum_plan* pl, double ln_k0) {
    pl->moments_ok       = false;
    const SmoothTable* t = pl->smooth;
    const int          F = pl->frac + 8;
    if (pl->nbins < 1 || F > 30) {
      return RG_OK;
    }
    std::vector<int64_t> tb(pl->nbins);
    std::vector<double>  eps(pl->nbins);
    std::vector<int4>    binfo(pl->nbins, make_int4(0, 0, 0, 0));
    int64_t tmin = std::numeric_limits<int64_t>::max(), tmax = std::numeric_limits<int64_t>::min();
    for (int b = 0; b < pl->nbins; ++b) {
      const double tt = (std::log(static_cast<double>(pl->h_bins[b])) - ln_k0 - t->ln_xmin) / t->dln;
      tb[b]           = std::llround(tt);
      eps[b]          = tt - static_cast<double>(tb[b]);
      tmin            = std::min(tmin, tb[b]);
      tmax            = std::max(tmax, tb[b]);
    }
    for (int b = 0; b < pl->nbins; ++b) {
      const float e32 = static_cast<float>(eps[b]);
      int         ebits;
      std::memcpy(&ebits, &e32, sizeof(ebits));
      binfo[b] = make_int4(static_cast<int>(tmax - tb[b]), ebits, 0, 1);
    }
    const int64_t cells = (tmax - tmin) + t->nseg;
    if (cells > (int64_t(1) << 24)) {
      return RG_OK;
    }
    pl->sm_pmin      = tmin << F;
    pl->sm_pmax      = tmax << F;
    pl->mom_L        = static_cast<int64_t>(t->nseg) << F;
    pl->sm_cells     = static_cast<int>(cells);
    pl->hist_per_seg = cells * kSub * 2; // double2 entries: kSub x 4 doubles per cell
    RG_CUDA_TRY(cudaMalloc(&pl->d_binfo, sizeof(int4) * binfo.size()));
    RG_CUDA_TRY(cudaMemcpy(pl->d_binfo, binfo.data(), sizeof(int4) * binfo.size(), cudaMemcpyHostToDevice));
    RG_TRY(fixed_log_prepare(pl, F, t->dln));
    if (pl->log_fx < 1) {
      return RG_OK; // no spacing of units fits (never for these tables); the fused kernels serve the plan
    }
    pl->moments_ok = true;
    return RG_OK;
  }

  // Per-(segment, cell) scratch for at least `entries` (segment, cell) pairs.
  int smooth_reserve_cells(rg_spectrum_plan* pl, size_t entries) {
    if (entries > pl->cells_cap) {
      cudaFree(pl->d_cells);
      pl->d_cells   = nullptr;
      pl->cells_cap = 0;
      RG_CUDA_TRY(cudaMalloc(&pl->d_cells, sizeof(float4) * entries));
      pl->cells_cap = entries;
    }
    return RG_OK;
  }

  int smooth_moments_deposit(rg_spectrum_plan* pl, const float* const comp[kComps], const int64_t* d_off, int64_t n,
                             int nseg, cudaStream_t s, uint2* place) {
    if (n == 0 && !d_off) {
      return moments_clear_sums(pl, s);
    }
    SmoothMomParams m;
    fill_smooth_params(pl, comp, d_off, n, nseg, m);
    m.run = run_sums(pl, d_off ? nseg : 1);
    DeviceContext* ctx = nullptr;
    RG_TRY(context(&ctx));
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
      m.place        = d_off || !place ? nullptr : place + w;
      const int grid = pair_grid(n, w, ctx->sms, kSmBlocksPerSM);
      if (m.fp.has_e) {
        if (d_off) {
          smooth_deposit_kernel<true, true><<<grid, kPairThreads, 0, s>>>(m);
        } else {
          smooth_deposit_kernel<true, false><<<grid, kPairThreads, 0, s>>>(m);
        }
      } else if (d_off) {
        smooth_deposit_kernel<false, true><<<grid, kPairThreads, 0, s>>>(m);
      } else {
        smooth_deposit_kernel<false, false><<<grid, kPairThreads, 0, s>>>(m);
      }
    }
    RG_CUDA_TRY(cudaGetLastError());
    if (pl->timing) {
      RG_CUDA_TRY(cudaEventRecord(ev.second, s));
      pl->ev_used.push_back(ev);
    }
    return RG_OK;
  }

  int smooth_moments_finish(rg_spectrum_plan* pl, int nseg, float* out, cudaStream_t s) {
    SmoothFinishParams r {};
    r.hist       = reinterpret_cast<double*>(pl->d_hist);
    r.nc         = pl->sm_cells;
    r.binfo      = pl->d_binfo;
    r.coef       = pl->smooth->d_coef;
    r.nseg_tab   = pl->smooth->nseg;
    r.nbins      = pl->nbins;
    r.ebins      = pl->d_ebins;
    r.status     = pl->d_status;
    r.acc        = pl->d_msum;
    r.acc_stride = pl->nslices * kSliceBins;
    r.done       = reinterpret_cast<unsigned*>(pl->d_msum + pl->msum_cap * kSliceBins);
    r.out        = out;
    r.nz         = negative_zeros();
    static std::atomic<uint64_t> configured { 0 };
    RG_CUDA_TRY(ensure_max_dynamic_smem(smooth_finish_kernel, static_cast<int>(sizeof(float4) * kSmoothMaxSegments), configured));
    smooth_finish_kernel<<<dim3((pl->sm_cells + kFinCells - 1) / kFinCells, nseg), kPairThreads,
                           sizeof(float4) * pl->smooth->nseg, s>>>(r);
    RG_CUDA_TRY(cudaGetLastError());
    pl->hist_dirty = pl->hist_stays_dirty;
    return RG_OK;
  }

  // The adjoint through cell cubics: grad_out is nseg x nbins; gradients of the particles
  // [0, n) (one segment) or of the segments of d_off.
  int smooth_moments_adjoint(rg_spectrum_plan* pl, const float* const comp[kComps], const int64_t* d_off, int64_t n,
                             int nseg, const float* grad_out, float* gw, float* const gu[3], cudaStream_t s,
                             const uint2* place) {
    const int    nsg  = d_off ? nseg : 1;
    const size_t need = static_cast<size_t>(nsg) * pl->sm_cells;
    RG_TRY(smooth_reserve_cells(pl, need));
    SmoothAlphaParams a {};
    a.grad_out = grad_out;
    a.binfo    = pl->d_binfo;
    a.coef     = pl->smooth->d_coef;
    a.nseg_tab = pl->smooth->nseg;
    a.nbins    = pl->nbins;
    a.ebins    = pl->d_ebins;
    a.nc       = pl->sm_cells;
    a.alpha    = pl->d_cells;
    smooth_alpha_kernel<<<dim3((pl->sm_cells + kSmAlphaThreads / 32 - 1) / (kSmAlphaThreads / 32), nsg), kSmAlphaThreads, 0,
                          s>>>(a);
    RG_CUDA_TRY(cudaGetLastError());
    if (n == 0 && !d_off) {
      return RG_OK;
    }
    SmoothAdjParams x {};
    fill_smooth_params(pl, comp, d_off, n, nseg, x.m);
    x.alpha   = pl->d_cells;
    x.inv_dln = static_cast<float>(1.0 / pl->smooth->dln);
    DeviceContext* ctx = nullptr;
    RG_TRY(context(&ctx));
    for (int64_t w = 0; w < std::max<int64_t>(n, 1); w += kPairWindow) {
      fill_streams(pl, comp, d_off, n, nseg, w, x.m.in);
      const int grid = pair_grid(n, w, ctx->sms, kSmAdjBlocksPerSM);
      x.place        = d_off || !place ? nullptr : place + w;
      x.gw           = gw ? gw + w : nullptr;
      for (int d = 0; d < 3; ++d) {
        x.gu[d] = gu[d] ? gu[d] + w : nullptr;
      }
      if (x.place) {
        if (x.m.fp.has_e) {
          smooth_adjoint_kernel<true, false, true><<<grid, kPairThreads, 0, s>>>(x);
        } else {
          smooth_adjoint_kernel<false, false, true><<<grid, kPairThreads, 0, s>>>(x);
        }
      } else if (x.m.fp.has_e) {
        if (d_off) {
          smooth_adjoint_kernel<true, true, false><<<grid, kPairThreads, 0, s>>>(x);
        } else {
          smooth_adjoint_kernel<true, false, false><<<grid, kPairThreads, 0, s>>>(x);
        }
      } else if (d_off) {
        smooth_adjoint_kernel<false, true, false><<<grid, kPairThreads, 0, s>>>(x);
      } else {
        smooth_adjoint_kernel<false, false, false><<<grid, kPairThreads, 0, s>>>(x);
      }
    }
    RG_CUDA_TRY(cudaGetLastError());
    return RG_OK;
  }

} // namespace rg

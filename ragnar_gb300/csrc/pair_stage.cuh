// The particle stage of the moment spectra for two particles per thread.
//
// What bounds the deposits is instruction issue, so the FP32 arithmetic of two particles
// runs in packed instructions (fma/add/mul.rn.f32x2: one issue slot for two IEEE
// operations; measured beside integer work, 57 packed instructions per clock and SM
// against 53 single ones), and the logarithm is taken from a table in the coordinate's own
// fixed-point units:
//   X = G W = 2^(E - 127) m,  c = 1 / m cut to 11 fraction bits,
//   r = m c - 1 (exact in FP32: a multiple of 2^-34 below 2^-10),
//   ln X = (E - 127) ln 2 - ln c + r - r^2/2 + r^3/3 + (low part of m) c,
// with ln c from a table of 64-bit integers indexed by c's own bits, so the
// reciprocal may be the hardware's approximate one.  The remainder's error is below 2^-41
// (r^4/4), a hundredth of the coordinate's unit.
//
// Every operation whose rounding error is taken is the IEEE operation written, and a particle whose
// X is not a normal float (u parallel to B, no field, overflow, NaN) takes the scalar
// stage instead.
#pragma once

#include "moments_common.cuh"
#include "spectrum_plan.hpp"

#include <algorithm>

namespace rg {

  // ---- asynchronous copies global -> shared ------------------------------------------------
  // 16 bytes, both addresses aligned to them; a thread's copies complete in the order of its commits.
  __device__ __forceinline__ void copy16(uint32_t dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
  }

  __device__ __forceinline__ void copies_commit() {
    asm volatile("cp.async.commit_group;" ::: "memory");
  }

  template <int kPending>
  __device__ __forceinline__ void copies_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(kPending) : "memory");
  }

  // ---- packed FP32 pairs ---------------------------------------------------------------
  struct f2 {
    unsigned long long v;
  };

  __device__ __forceinline__ f2 pack2(float lo, float hi) {
    f2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(lo), "f"(hi));
    return r;
  }

  __device__ __forceinline__ void unpack2(f2 a, float& lo, float& hi) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(a.v));
  }

  __device__ __forceinline__ f2 set2(float x) {
    return pack2(x, x);
  }

  __device__ __forceinline__ f2 add2(f2 a, f2 b) {
    f2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
  }

  // The compiler may contract a packed product and a packed sum into an fma, .rn or not (measured:
  // 489284 of 1048576 sums of three squares differ from the separately rounded ones).  A product whose
  // own rounding a sum takes for granted is a product2.
  __device__ __forceinline__ f2 mul2(f2 a, f2 b) {
    f2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
  }

  __device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) {
    f2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
    return r;
  }

  // a b, rounded: nz is a pair of -0 that the kernel gets as a parameter, so that the compiler sees an
  // fma with an unknown addend and has nothing to contract.
  __device__ __forceinline__ f2 product2(f2 a, f2 b, f2 nz) {
    return fma2(a, b, nz);
  }

  inline f2 negative_zeros() {
    return { 0x8000000080000000ull };
  }

  // a - b: one rounding, as a subtraction
  __device__ __forceinline__ f2 sub2(f2 a, f2 b) {
    return fma2(b, set2(-1.0f), a);
  }

  struct ff2 {
    f2 hi, lo;
  };

  __device__ __forceinline__ ff2 two_sum2(f2 a, f2 b) {
    const f2 s  = add2(a, b);
    const f2 bb = sub2(s, a);
    return { s, add2(sub2(a, sub2(s, bb)), sub2(b, bb)) };
  }

  __device__ __forceinline__ ff2 fast_two_sum2(f2 a, f2 b) { // |a| >= |b|
    const f2 s = add2(a, b);
    return { s, sub2(b, sub2(s, a)) };
  }

  __device__ __forceinline__ ff2 ff_add2(ff2 a, ff2 b) {
    const ff2 s = two_sum2(a.hi, b.hi);
    return fast_two_sum2(s.hi, add2(s.lo, add2(a.lo, b.lo)));
  }

  __device__ __forceinline__ f2 neg2(f2 a) {
    return mul2(a, set2(-1.0f));
  }

  // ---- kinematics ------------------------------------------------------------------------
  // G = 1 + u^2 and W = |gamma E + u x B|^2 - (u.E)^2 of two particles: G = Gh - nGl, W = Wh + Wl
  // (relative error ~2^-44; the high parts are within a few ulp of the sums, not normalised).
  struct Kin2 {
    f2 Gh, nGl, Wh, Wl;
  };

  // a b - c d with na = -a and nc = -c, as a normalised pair: when the products nearly cancel,
  // their remainders carry the whole value.
  __device__ __forceinline__ ff2 diff_of_products2(f2 a, f2 na, f2 b, f2 c, f2 nc, f2 d, f2 nz) {
    const f2  p = product2(a, b, nz), q = product2(nc, d, nz);
    const f2  e = add2(fma2(na, b, p), fma2(c, d, q)); // -(remainder of p + remainder of q)
    const ff2 r = two_sum2(p, q);
    return fast_two_sum2(r.hi, sub2(r.lo, e));
  }

  // a^2 of a pair: hi = a.hi^2 and the negative of everything below it
  __device__ __forceinline__ void square2(ff2 a, f2& hi, f2& nlo, f2 nz) {
    hi  = product2(a.hi, a.hi, nz);
    nlo = fma2(mul2(a.hi, set2(-2.0f)), a.lo, fma2(neg2(a.hi), a.hi, hi));
  }

  template <bool kE>
  __device__ __forceinline__ Kin2 kinematics2(const f2 (&v)[kComps], f2 nz) {
    const f2 ux = v[0], uy = v[1], uz = v[2];
    const f2 nx = neg2(ux), ny = neg2(uy), mz = neg2(uz);
    Kin2     k;
    {
      const f2  x2 = product2(ux, ux, nz), y2 = product2(uy, uy, nz), z2 = product2(uz, uz, nz);
      const f2  e  = add2(add2(fma2(nx, ux, x2), fma2(ny, uy, y2)), fma2(mz, uz, z2));
      const ff2 s  = two_sum2(x2, y2);
      const ff2 t  = two_sum2(s.hi, z2);
      const ff2 g  = two_sum2(set2(1.0f), t.hi);
      k.Gh         = g.hi;
      k.nGl        = sub2(e, add2(add2(s.lo, t.lo), g.lo));
    }
    const f2 bx = v[6], by = v[7], bz = v[8];
    ff2      cx = diff_of_products2(uy, ny, bz, uz, mz, by, nz);
    ff2      cy = diff_of_products2(uz, mz, bx, ux, nx, bz, nz);
    ff2      cz = diff_of_products2(ux, nx, by, uy, ny, bx, nz);
    if (!kE) {
      f2 hx, hy, hz, lx, ly, lz;
      square2(cx, hx, lx, nz);
      square2(cy, hy, ly, nz);
      square2(cz, hz, lz, nz);
      const ff2 s = two_sum2(hx, hy);
      const ff2 t = two_sum2(s.hi, hz);
      k.Wh        = t.hi;
      k.Wl        = sub2(add2(s.lo, t.lo), add2(add2(lx, ly), lz));
      return k;
    }
    const f2 ex = v[3], ey = v[4], ez = v[5];
    // gamma = sqrt(G): g = Gh y with y ~ 1 / sqrt(Gh), and the remainder (G - g^2) y / 2
    float g0, g1;
    unpack2(k.Gh, g0, g1);
    const f2 y  = pack2(rsqrtf(g0), rsqrtf(g1));
    const f2 gh = mul2(k.Gh, y);
    const f2 gl = mul2(sub2(fma2(neg2(gh), gh, k.Gh), k.nGl), mul2(y, set2(0.5f)));
    const f2 ng = neg2(gh);
    auto     term = [&](f2 e, ff2 c) { // gamma e + c
      const f2 p = product2(gh, e, nz);
      return ff_add2(ff2 { p, sub2(mul2(gl, e), fma2(ng, e, p)) }, c);
    };
    cx = term(ex, cx);
    cy = term(ey, cy);
    cz = term(ez, cz);
    // u.E
    const f2  px = product2(ux, ex, nz), py = product2(uy, ey, nz), pz = product2(uz, ez, nz);
    const f2  e  = add2(add2(fma2(nx, ex, px), fma2(ny, ey, py)), fma2(mz, ez, pz));
    const ff2 s  = two_sum2(px, py);
    const ff2 t  = two_sum2(s.hi, pz);
    const ff2 d  = fast_two_sum2(t.hi, sub2(add2(s.lo, t.lo), e));
    f2        hx, hy, hz, hd, lx, ly, lz, ld;
    square2(cx, hx, lx, nz);
    square2(cy, hy, ly, nz);
    square2(cz, hz, lz, nz);
    square2(d, hd, ld, nz);
    const ff2 a = two_sum2(hx, hy);
    const ff2 b = two_sum2(a.hi, hz);
    const ff2 w = two_sum2(b.hi, neg2(hd));
    const ff2 W = fast_two_sum2(w.hi, add2(add2(add2(a.lo, b.lo), w.lo), sub2(ld, add2(add2(lx, ly), lz))));
    k.Wh        = W.hi;
    k.Wl        = W.lo;
    return k;
  }

  // ---- table coordinate and amplitude ------------------------------------------------------

  // c = 1 / m by the hardware, cut to 11 fraction bits: (0.5, 1], or an ulp below 0.5 for m next to 2.
  // Its table index is 11 bits of its bit pattern: the lowest exponent bit and ten mantissa bits,
  // so c in [0.5, 1) takes entries 0 .. 1023, c = 1 entry 1024, and c just below 0.5 the last
  // one; no value, not even NaN, indexes past the table.
  constexpr int kLogShift   = 13;
  constexpr int kLogEntries = 2048;

  // Fixed-point constants of a plan's coordinate: units of 2^-(F + fx) table segments, fx chosen
  // so that S 2^-10 stays below 2^31 (fixed_log_prepare).
  struct LogParams {
    float          Sh, Sl; // S = 2^(F + fx) / (2 dln) as a double-float
    int64_t        Cfx;    // round(S ln 2)
    int            fx;
    const int64_t* table;  // round(S ln c), kLogEntries; then the constants of stand_in
    f2             nz;     // of product2
  };

  inline void fill_log_params(const rg_spectrum_plan* pl, LogParams& g) {
    g.Sh    = pl->log_Sh;
    g.Sl    = pl->log_Sl;
    g.Cfx   = pl->log_Cfx;
    g.fx    = pl->log_fx;
    g.table = pl->d_logt;
    g.nz    = negative_zeros();
  }

  // What a deposit reads, with a stride of 0, for a particle stream that is not given: zero field,
  // unit weight; kStandIn floats, as the second of a thread's two loads is 256 floats further.
  constexpr int kStandIn = 257;

  inline const float* stand_in(const rg_spectrum_plan* pl, int comp) {
    return reinterpret_cast<const float*>(pl->d_logt + kLogEntries) + (comp == 9 ? kStandIn : 0);
  }

  // Stages the log table, with everything of Y that does not depend on the particle added:
  // 2^fx Pmax, half a unit for the rounding, the exponent's bias, and -2^31 for place2's offset.
  __device__ __forceinline__ void stage_log_table(const LogParams& g, int fx, int64_t Pmax, int64_t* logt, int threads) {
    const int64_t base = (Pmax << fx) + ((int64_t(1) << (fx - 1)) - 1) + 127 * g.Cfx - (int64_t(1) << 31);
    for (int i = threadIdx.x; i < kLogEntries; i += threads) {
      logt[i] = g.table[i] + base;
    }
  }

  // Whether a particle of amplitude A adds anything (0 does not, nor do infinities and NaN, as in
  // the scalar stage).
  __device__ __forceinline__ bool emits(float A) {
    return (__float_as_uint(A) << 1) - 1u < 0xfeffffffu;
  }

  // Y = 2^fx (Pmax - Q) before rounding to whole units: cell and low part of R = Pmax - Q are
  // Y >> (F + fx) and (Y >> fx) mod 2^F, and a particle outside every bin's table range lands
  // at a negative Y or past the last cell.  A: the amplitude w chiR / B0 (see emits).
  struct Place2 {
    int64_t Y[2];
    float   A[2];
  };

  // The scalar stage, for the particles the packed one leaves out (a call, not inlined: rare).
  static __device__ __noinline__ int64_t scalar_place(const float (&v)[kComps], const FusedParams& p, int fx, int64_t Pmin,
                                               int64_t Pmax, int64_t L, float& A) {
    int64_t Q = 0;
    if (!moment_particle_stage(v, p, Pmin, Pmax, L, Q, A)) {
      A = 0.0f;
      return -1;
    }
    return (Pmax - Q) << fx;
  }

  template <bool kE>
  __device__ __forceinline__ Place2 place2(const f2 (&v)[kComps], const FusedParams& p, const LogParams& g,
                                           const int64_t* logt, int64_t Pmin, int64_t Pmax, int64_t L) {
    const Kin2 k = kinematics2<kE>(v, g.nz);
    // X = G W = xh - nxl
    const f2 nG  = neg2(k.Gh);
    const f2 xh  = mul2(k.Gh, k.Wh);
    const f2 nxl = fma2(k.nGl, k.Wh, fma2(nG, k.Wl, fma2(nG, k.Wh, xh)));
    float    x[2];
    unpack2(xh, x[0], x[1]);
    uint32_t E[2];
    float    sc[2], y[2];
    bool     normal[2];
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const uint32_t b = __float_as_uint(x[j]);
      normal[j]        = x[j] >= 1.17549435e-38f && x[j] < 1.7014118e38f; // false for NaN
      E[j]             = b >> 23;
      sc[j]            = __uint_as_float(0x7f000000u - (b & 0x7f800000u)); // 2^(127 - E)
      asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y[j]) : "f"(x[j]));
    }
    const f2 sc2 = pack2(sc[0], sc[1]);
    const f2 m2  = mul2(xh, sc2);
    float    m[2], c[2];
    int64_t  T[2];
    unpack2(m2, m[0], m[1]);
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const uint32_t cb = __float_as_uint(rcp_approx(m[j]));
      c[j]              = __uint_as_float(cb & ~((1u << kLogShift) - 1u));
      T[j]              = logt[(cb >> kLogShift) & (kLogEntries - 1)];
    }
    const f2 c2  = pack2(c[0], c[1]);
    const f2 r   = fma2(m2, c2, set2(-1.0f));
    const f2 np  = fma2(mul2(r, r), fma2(r, set2(-0.33333334f), set2(0.5f)), mul2(mul2(nxl, sc2), c2));
    const f2 ph  = mul2(r, set2(g.Sh));
    const f2 npl = fma2(np, set2(g.Sh), fma2(r, set2(-g.Sl), fma2(r, set2(-g.Sh), ph)));
    float    h[2], nl[2];
    unpack2(ph, h[0], h[1]);
    unpack2(npl, nl[0], nl[1]);
    // chiR = W / sqrt(X) with y ~ 1 / sqrt(xh): s0 = Wh y, plus Wl y + s0 (1 - X y^2) / 2 and the
    // remainder of s0
    const f2 yy  = pack2(y[0], y[1]);
    const f2 nyy = neg2(yy);
    const f2 q   = mul2(xh, yy);
    const f2 mt  = fma2(nxl, yy, fma2(xh, nyy, q)); // -(low part of X y + remainder of q)
    const f2 e   = fma2(mt, yy, fma2(q, nyy, set2(1.0f)));
    const f2 s0  = product2(k.Wh, yy, g.nz);
    const f2 u   = fma2(mul2(s0, set2(0.5f)), e, mul2(k.Wl, yy));
    const f2 chi = add2(s0, sub2(u, fma2(k.Wh, nyy, s0)));
    const f2 A   = mul2(mul2(chi, set2(p.amp)), v[9]);
    Place2   o;
    unpack2(A, o.A[0], o.A[1]);
    const uint32_t nlo = static_cast<uint32_t>(-g.Cfx), nhi = static_cast<uint32_t>(-g.Cfx >> 32);
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      // the int32 correction, offset by 2^31 to add as an unsigned number; E (-Cfx) modulo 2^64
      const uint32_t i = static_cast<uint32_t>(__float2int_rn(nl[j]) - __float2int_rn(h[j])) + 0x80000000u;
      uint64_t       Y = static_cast<uint64_t>(E[j]) * nlo + static_cast<uint64_t>(T[j]);
      Y += static_cast<uint64_t>(E[j] * nhi) << 32;
      o.Y[j] = static_cast<int64_t>(Y + i);
    }
    if (!(normal[0] && normal[1])) {
      float wh[2], wl[2];
      unpack2(k.Wh, wh[0], wh[1]);
      unpack2(k.Wl, wl[0], wl[1]);
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        if (normal[j]) {
          continue;
        }
        if (wh[j] == 0.0f && wl[j] == 0.0f) { // no emission: u parallel to B, or no field
          o.Y[j] = -1;
          o.A[j] = 0.0f;
          continue;
        }
        float s[kComps];
#pragma unroll
        for (int d = 0; d < kComps; ++d) {
          float lo, hi;
          unpack2(v[d], lo, hi);
          s[d] = j ? hi : lo;
        }
        float a;
        o.Y[j] = scalar_place(s, p, g.fx, Pmin, Pmax, L, a);
        o.A[j] = a;
      }
    }
    return o;
  }

  // ---- particle streams, two particles per thread ------------------------------------------
  // What a kernel over pairs reads: the streams from the first particle of the launch's window of
  // at most kPairWindow particles (32-bit indices within it), and the segments.
  constexpr int     kPairThreads = 256;
  constexpr int     kPairChunk   = 2 * kPairThreads;   // particles per block and step
  constexpr int64_t kPairWindow  = int64_t(1) << 31;
  constexpr int     kPairSharedSeg = 1024;             // segment offsets staged in shared memory

  struct PairStreams {
    const float*   comp[kComps];   // a stand-in where a stream is not given
    uint32_t       stride[kComps]; // bytes between particles: 4, or 0 for a stand-in
    const int64_t* seg_off;        // nseg + 1 particle offsets (device), or null: particles [0, n)
    int            nseg;
    int64_t        n;              // stream length
    int64_t        window;         // the window's first particle
  };

  inline void fill_streams(const rg_spectrum_plan* pl, const float* const comp[kComps], const int64_t* d_off, int64_t n,
                           int nseg, int64_t window, PairStreams& p) {
    for (int c = 0; c < kComps; ++c) {
      p.comp[c]   = comp[c] ? comp[c] + window : stand_in(pl, c);
      p.stride[c] = comp[c] ? 4u : 0u;
    }
    p.seg_off = d_off;
    p.nseg    = d_off ? nseg : 1;
    p.n       = n;
    p.window  = window;
  }

  // Blocks over the window's particles, at most per_sm per SM.
  inline int pair_grid(int64_t n, int64_t window, int sms, int per_sm) {
    const int64_t steps = (std::min(n - window, kPairWindow) + kPairChunk - 1) / kPairChunk;
    return static_cast<int>(std::max<int64_t>(1, std::min<int64_t>(steps, static_cast<int64_t>(sms) * per_sm)));
  }

  // The finish kernel's bin sums and block counts, cleared by the deposit that comes before it on the
  // stream, whatever an earlier run left in them.
  struct RunSums {
    double*   sums;
    int64_t   nsums;
    unsigned* done;
    int64_t   ndone;
  };

  inline RunSums run_sums(const rg_spectrum_plan* pl, int nseg) {
    const int64_t rows = static_cast<int64_t>(nseg) * pl->nslices;
    return { pl->d_msum, rows * kSliceBins, reinterpret_cast<unsigned*>(pl->d_msum + pl->msum_cap * kSliceBins), rows };
  }

  __device__ __forceinline__ void clear_run_sums(const RunSums& r) {
    const int64_t step = static_cast<int64_t>(gridDim.x) * gridDim.y * kPairThreads;
    const int64_t i0   = (static_cast<int64_t>(blockIdx.y) * gridDim.x + blockIdx.x) * kPairThreads + threadIdx.x;
    for (int64_t i = i0; i < r.nsums; i += step) {
      r.sums[i] = 0.0;
    }
    for (int64_t i = i0; i < r.ndone; i += step) {
      r.done[i] = 0u;
    }
  }

  // Stages the segments' offsets, clamped to the window and relative to its start; false for the
  // whole block if they decrease or leave [0, n], or if the status word is set.
  template <bool kSeg>
  __device__ __forceinline__ bool stage_segments(const PairStreams& p, unsigned* status, uint32_t* soff) {
    const int64_t w0 = p.window, w1 = min(p.n, w0 + kPairWindow);
    bool          bad = false;
    if (kSeg) {
      for (int i = threadIdx.x; i <= p.nseg; i += kPairThreads) {
        const int64_t o = p.seg_off[i];
        bad             = bad || o < 0 || o > p.n || (i > 0 && o < p.seg_off[i - 1]);
        soff[i]         = static_cast<uint32_t>(max(min(o, w1), w0) - w0);
      }
    }
    if (__syncthreads_or(bad)) {
      if (threadIdx.x == 0 && blockIdx.x == 0 && blockIdx.y == 0) {
        atomicOr(status, kDevBadOffsets);
      }
      return false;
    }
    return !__syncthreads_or(*status != kDevOk);
  }

  // Particles base + thread and base + thread + 256 (coalesced whatever the streams' alignment).
  // Past the end the last particle again, to be dropped by its index; nothing from a base past it.
  template <bool kE>
  __device__ __forceinline__ void load_pair(const PairStreams& p, uint32_t base, uint32_t last, float2 (&to)[kComps]) {
    if (base + kPairChunk <= last) {
#pragma unroll
      for (int c = 0; c < kComps; ++c) {
        if (kE || c < 3 || c >= 6) {
          const float* q = reinterpret_cast<const float*>(reinterpret_cast<const char*>(p.comp[c]) +
                                                          static_cast<uint64_t>(base + threadIdx.x) * p.stride[c]);
          to[c].x        = __ldg(q);
          to[c].y        = __ldg(q + kPairThreads);
        }
      }
    } else if (base < last) {
      const uint32_t i0 = min(base + threadIdx.x, last - 1), i1 = min(base + threadIdx.x + kPairThreads, last - 1);
#pragma unroll
      for (int c = 0; c < kComps; ++c) {
        if (kE || c < 3 || c >= 6) {
          const char* q = reinterpret_cast<const char*>(p.comp[c]);
          to[c].x       = __ldg(reinterpret_cast<const float*>(q + static_cast<uint64_t>(i0) * p.stride[c]));
          to[c].y       = __ldg(reinterpret_cast<const float*>(q + static_cast<uint64_t>(i1) * p.stride[c]));
        }
      }
    }
  }

  template <bool kE>
  __device__ __forceinline__ void to_pairs(const float2 (&from)[kComps], f2 (&v)[kComps]) {
#pragma unroll
    for (int c = 0; c < kComps; ++c) {
      v[c] = (kE || c < 3 || c >= 6) ? pack2(from[c].x, from[c].y) : set2(0.0f);
    }
  }

  // FP64 add to global memory where `on`, without a branch.
  __device__ __forceinline__ void red_add_if(bool on, double* p, double v) {
    asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %2, 0;\n\t@q red.global.add.f64 [%0], %1;\n\t}" ::"l"(p), "d"(v),
                 "r"(static_cast<uint32_t>(on))
                 : "memory");
  }

  constexpr uint32_t kNoEntry = 0xffffffffu;

  // d 2^-k as (hi, lo): the top 24 significant bits cut, then the 29 below; 0 when d 2^-k < 2^-126
  // (GB300's FP64 pipe would take longer over the subtraction d - hi than these integer steps).
  __device__ __forceinline__ float2 split_double(double d, int k) {
    const uint32_t h = static_cast<uint32_t>(__double2hiint(d)), l = static_cast<uint32_t>(__double2loint(d));
    const int      e = static_cast<int>((h >> 20) & 0x7ffu) - 1023 + 127 - k; // biased FP32 exponent
    const uint32_t sign = h & 0x80000000u;
    float2         r;
    r.x = __uint_as_float(sign | (static_cast<uint32_t>(e) << 23) | (__funnelshift_l(l, h, 3) & 0x7fffffu));
    r.y = static_cast<float>(l & 0x1fffffffu) * __uint_as_float(sign | (static_cast<uint32_t>(e - 52) << 23));
    r.y = e > 52 ? r.y : 0.0f;
    return e >= 1 ? r : make_float2(0.0f, 0.0f);
  }

  __device__ __forceinline__ ff2 ff_mul2(ff2 a, ff2 b, f2 nz) {
    const f2 p = product2(a.hi, b.hi, nz);
    const f2 e = sub2(fma2(a.hi, b.lo, mul2(a.lo, b.hi)), fma2(neg2(a.hi), b.hi, p));
    return fast_two_sum2(p, e);
  }

} // namespace rg

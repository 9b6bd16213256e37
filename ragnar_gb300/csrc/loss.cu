// The misfit of spectra, mean((ln S - ln T)^2) over the bins above a floor of both peaks, with what
// its derivatives need.
//
// Written as tensor operations it takes about 20 launches forward and 15 backward on a few hundred
// values, and the host's time for them is most of a training step on small inputs.  Here a
// spectrum of up to kLossOneBlock values takes one launch and larger sets three.
//
// With d = ln S - ln T and m the c values that count, the outputs are the loss, r = m 2 d / (c S) (the
// gradient) and a = m / S; dr/dS = 2 a^2 / c - r a and da/dS = -a^2 give every higher derivative from the
// same two arrays.
//
// Bound by launch and reduction latency.  GB300's FP64 adds come at 2 lanes a clock, so threads and
// warps sum in double-floats and only one warp a block in FP64: 512 values 9.9 -> 5.0 us, the finish of
// 1024 x 512 values 9.1 -> 6.5 us.  A training step of 2e4 particles falls from 744 to 394 us (what is
// left is the autograd engine's and the host's), a fit of 1024 distributions from 674 to 345 us.
#include "rg_common.cuh"
#include "rg_internal.hpp"

#include <algorithm>

namespace rg {

  namespace {

    constexpr int     kLossThreads   = 1024;
    constexpr int64_t kLossOneBlock  = 8192; // values of the one-block kernel (eight a thread)
    constexpr int     kLossPerThread = 4;    // values a thread of the larger grids, at least

    struct LossParams {
      const float* S;
      const float* T;
      int64_t      n;
      float        floor;
      float*       r;
      float*       a;
      float*       loss;
      float*       inv_count;
      float2*      peak; // [grid] block maxima
      double2*     sums; // [grid] (sum of d^2, count) of a block
      int          grid;
    };

    // The larger value; NaN if either is (as the peak of a spectrum with NaN).
    __device__ __forceinline__ float larger(float a, float b) {
      return a > b || a != a ? a : b;
    }

    __device__ __forceinline__ float2 block_peak(float2 v, float2* shared) {
      for (int o = 16; o > 0; o >>= 1) {
        v.x = larger(v.x, __shfl_xor_sync(0xffffffffu, v.x, o));
        v.y = larger(v.y, __shfl_xor_sync(0xffffffffu, v.y, o));
      }
      if ((threadIdx.x & 31) == 0) {
        shared[threadIdx.x >> 5] = v;
      }
      __syncthreads();
      v = shared[threadIdx.x & 31]; // kLossThreads / 32 = 32 entries
      for (int o = 16; o > 0; o >>= 1) {
        v.x = larger(v.x, __shfl_xor_sync(0xffffffffu, v.x, o));
        v.y = larger(v.y, __shfl_xor_sync(0xffffffffu, v.y, o));
      }
      return v;
    }

    struct Sum {
      ff       v;
      unsigned count;
    };

    // v over a warp of FP64 pairs, the same in every lane
    __device__ __forceinline__ double2 warp_sum(double2 v) {
      for (int o = 16; o > 0; o >>= 1) {
        v.x += __shfl_xor_sync(0xffffffffu, v.x, o);
        v.y += __shfl_xor_sync(0xffffffffu, v.y, o);
      }
      return v;
    }

    // Of a block's sums; only warp 0 has the result.
    __device__ __forceinline__ double2 block_sum(Sum s, float2* part, unsigned* counts) {
      for (int o = 16; o > 0; o >>= 1) {
        s.v = ff_add(s.v, ff { __shfl_xor_sync(0xffffffffu, s.v.hi, o), __shfl_xor_sync(0xffffffffu, s.v.lo, o) });
      }
      s.count = __reduce_add_sync(0xffffffffu, s.count);
      if ((threadIdx.x & 31) == 0) {
        part[threadIdx.x >> 5]   = make_float2(s.v.hi, s.v.lo);
        counts[threadIdx.x >> 5] = s.count;
      }
      __syncthreads();
      if (threadIdx.x >= 32) {
        return make_double2(0.0, 0.0);
      }
      const float2 p = part[threadIdx.x];
      // an infinite or NaN sum's low part is NaN
      return warp_sum(make_double2(static_cast<double>(p.x) + (isfinite(p.x) ? static_cast<double>(p.y) : 0.0),
                                   static_cast<double>(counts[threadIdx.x])));
    }

    // Peaks of the values i, i + step, ...
    __device__ __forceinline__ float2 peaks(const LossParams& p, int64_t i, int64_t step) {
      const float low = __int_as_float(0xff800000);
      float2      v   = make_float2(low, low);
      for (; i < p.n; i += step) {
        v.x = larger(v.x, p.S[i]);
        v.y = larger(v.y, p.T[i]);
      }
      return v;
    }

    // d (0 where a value does not count) and a of the same values, and their part of the sum and the count.
    __device__ __forceinline__ Sum terms(const LossParams& p, float2 peak, int64_t i, int64_t step) {
      const float lowS = __fmul_rn(p.floor, peak.x), lowT = __fmul_rn(p.floor, peak.y);
      Sum         t { { 0.0f, 0.0f }, 0u };
      for (; i < p.n; i += step) {
        const float s = p.S[i], y = p.T[i];
        const bool  m = s > lowS && y > lowT;
        const float d = m ? logf(s) - logf(y) : 0.0f;
        p.r[i]        = d;
        p.a[i]        = m ? __frcp_rn(s) : 0.0f;
        t.v           = ff_add(t.v, two_prod(d, d));
        t.count += m ? 1u : 0u;
      }
      return t;
    }

    // The loss and 1 / c, and r = (2 d / c) / S from the d that terms left in its place: 2 d / S itself is
    // above the float range for spectra near its lower end.
    __device__ __forceinline__ void finish(const LossParams& p, double2 t, float* inv, int64_t i, int64_t step) {
      if (threadIdx.x == 0) {
        const double count = fmax(t.y, 1.0);
        *inv               = static_cast<float>(1.0 / count);
        if (blockIdx.x == 0) {
          *p.loss      = static_cast<float>(t.x / count);
          *p.inv_count = *inv;
        }
      }
      __syncthreads();
      for (; i < p.n; i += step) {
        const float d = p.r[i];
        p.r[i]        = d != 0.0f ? __fdiv_rn(__fmul_rn(d + d, *inv), p.S[i]) : 0.0f;
      }
    }

    __global__ void __launch_bounds__(kLossThreads) loss_one_kernel(const __grid_constant__ LossParams p) {
      __shared__ float2   part[32];
      __shared__ float2   peak[32];
      __shared__ unsigned counts[32];
      __shared__ float    inv;
      const float2        top = block_peak(peaks(p, threadIdx.x, kLossThreads), peak);
      finish(p, block_sum(terms(p, top, threadIdx.x, kLossThreads), part, counts), &inv, threadIdx.x, kLossThreads);
    }

    __global__ void __launch_bounds__(kLossThreads) loss_peak_kernel(const __grid_constant__ LossParams p) {
      __shared__ float2 sp[32];
      const int64_t     step = static_cast<int64_t>(gridDim.x) * kLossThreads;
      const float2      peak = block_peak(peaks(p, static_cast<int64_t>(blockIdx.x) * kLossThreads + threadIdx.x, step), sp);
      if (threadIdx.x == 0) {
        p.peak[blockIdx.x] = peak;
      }
    }

    __global__ void __launch_bounds__(kLossThreads) loss_terms_kernel(const __grid_constant__ LossParams p) {
      __shared__ float2   part[32];
      __shared__ float2   peak[32];
      __shared__ unsigned counts[32];
      const float         low  = __int_as_float(0xff800000);
      const int64_t       step = static_cast<int64_t>(gridDim.x) * kLossThreads;
      const float2 top = block_peak(static_cast<int>(threadIdx.x) < p.grid ? p.peak[threadIdx.x] : make_float2(low, low), peak);
      const double2 t = block_sum(terms(p, top, static_cast<int64_t>(blockIdx.x) * kLossThreads + threadIdx.x, step), part, counts);
      if (threadIdx.x == 0) {
        p.sums[blockIdx.x] = t;
      }
    }

    __global__ void __launch_bounds__(kLossThreads) loss_finish_kernel(const __grid_constant__ LossParams p) {
      __shared__ float inv;
      double2          t = make_double2(0.0, 0.0);
      if (threadIdx.x < 32) {
        for (int k = threadIdx.x; k < p.grid; k += 32) {
          const double2 v = p.sums[k];
          t.x += v.x;
          t.y += v.y;
        }
        t = warp_sum(t);
      }
      finish(p, t, &inv, static_cast<int64_t>(blockIdx.x) * kLossThreads + threadIdx.x,
             static_cast<int64_t>(gridDim.x) * kLossThreads);
    }

  } // namespace

} // namespace rg

extern "C" {

int rg_log_mse(const float* S, const float* T, int64_t n, float floor, float* r, float* a, float* loss,
               float* inv_count, void* stream) {
  rg::NvtxRange nvtx_range("LogMse");
  rg::clear_error();
  if (n < 1 || !S || !T || !r || !a || !loss || !inv_count) {
    return rg::set_error(RG_ERR_ARGUMENT, "rg_log_mse: bad arguments");
  }
  auto           s = static_cast<cudaStream_t>(stream);
  rg::LossParams p {};
  p.S         = S;
  p.T         = T;
  p.n         = n;
  p.floor     = floor;
  p.r         = r;
  p.a         = a;
  p.loss      = loss;
  p.inv_count = inv_count;
  if (n <= rg::kLossOneBlock) {
    rg::loss_one_kernel<<<1, rg::kLossThreads, 0, s>>>(p);
    RG_CUDA_TRY(cudaGetLastError());
    return RG_OK;
  }
  rg::DeviceContext* ctx = nullptr;
  RG_TRY(rg::context(&ctx));
  // two blocks an SM, at most as many as one block reads back (kLossThreads)
  const int64_t per = static_cast<int64_t>(rg::kLossThreads) * rg::kLossPerThread;
  p.grid = static_cast<int>(std::min<int64_t>((n + per - 1) / per, std::min(2 * ctx->sms, rg::kLossThreads)));
  unsigned char* buf = nullptr;
  RG_TRY(rg::scratch_alloc(reinterpret_cast<void**>(&buf), (sizeof(double2) + sizeof(float2)) * p.grid, s));
  p.sums = reinterpret_cast<double2*>(buf);
  p.peak = reinterpret_cast<float2*>(buf + sizeof(double2) * p.grid);
  rg::loss_peak_kernel<<<p.grid, rg::kLossThreads, 0, s>>>(p);
  rg::loss_terms_kernel<<<p.grid, rg::kLossThreads, 0, s>>>(p);
  rg::loss_finish_kernel<<<p.grid, rg::kLossThreads, 0, s>>>(p);
  const cudaError_t e = cudaGetLastError();
  const cudaError_t f = cudaFreeAsync(buf, s);
  if (e != cudaSuccess) {
    return rg::cuda_error(e, "rg_log_mse launch");
  }
  RG_CUDA_TRY(f);
  return RG_OK;
}

} // extern "C"

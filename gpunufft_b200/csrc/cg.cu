// Vector updates of the conjugate-gradient solve (cg_sense_2d.m:40-108 of
// the upstream demos), fused: per iteration one pass for <p, M p>, one for
// x, r and ||r||^2, one for the next direction, every scalar staying on the
// device.
//
// Bound by launch latency at 2-D sizes: 256^2 pixels on a B200, the eleven
// elementwise and reduction launches of a composed iteration took 33 us of
// device time and as many host calls; these three take 15 us.
#include <algorithm>

#include "capi.hpp"
#include "cplx.cuh"
#include "devutil.hpp"
#include "planview.hpp"

namespace gnufft
{
namespace
{
constexpr int kCgThreads = 256;
constexpr int kCgMaxBlocks = 444;

struct CgWork
{
  float rr;    // ||r||^2 (first word: read by the caller)
  float beta;  // ||r_new||^2 / ||r||^2
  float2 a;    // ||r||^2 / <p, M p>
  unsigned done;
  unsigned pad[3];
  double2 partial[kCgMaxBlocks];
};
static_assert(sizeof(CgWork) <= GNUFFT_CG_WORK_BYTES, "work buffer size");

// Block sum in a fixed order; valid in thread 0.
__device__ __forceinline__ double2 block_sum(double2 v)
{
  __shared__ double2 s[kCgThreads / 32];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
  {
    v.x += __shfl_down_sync(0xffffffffu, v.x, o);
    v.y += __shfl_down_sync(0xffffffffu, v.y, o);
  }
  __syncthreads();
  if ((threadIdx.x & 31) == 0)
    s[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x == 0)
    for (int i = 1; i < kCgThreads / 32; ++i)
    {
      v.x += s[i].x;
      v.y += s[i].y;
    }
  return v;
}

// The blocks' sums meet in the block that finishes last, which adds them in
// block order (the result does not depend on which block that is) and calls
// f(sum) in thread 0.
template <class F>
__device__ __forceinline__ void grid_sum(double2 v, CgWork *w, F f)
{
  __shared__ bool last;
  v = block_sum(v);
  if (threadIdx.x == 0)
  {
    w->partial[blockIdx.x] = v;
    __threadfence();
    last = atomicAdd(&w->done, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last)
    return;
  __threadfence();
  double2 t = make_double2(0.0, 0.0);
  for (unsigned i = threadIdx.x; i < gridDim.x; i += kCgThreads)
  {
    const volatile double2 *q = &w->partial[i];
    t.x += q->x;
    t.y += q->y;
  }
  t = block_sum(t);
  if (threadIdx.x == 0)
  {
    w->done = 0u;
    f(t);
  }
}

__global__ void __launch_bounds__(kCgThreads)
    k_cg_begin(const float2 *__restrict__ r, size_t n, CgWork *w)
{
  double2 s = make_double2(0.0, 0.0);
  for (size_t i = (size_t)blockIdx.x * kCgThreads + threadIdx.x; i < n;
       i += (size_t)gridDim.x * kCgThreads)
  {
    const float2 v = r[i];
    s.x += (double)v.x * v.x + (double)v.y * v.y;
  }
  grid_sum(s, w, [&](double2 t) { w->rr = (float)t.x; });
}

// a = rr / <p, q>, <p, q> = sum conj(p) q
__global__ void __launch_bounds__(kCgThreads)
    k_cg_dot(const float2 *__restrict__ p, const float2 *__restrict__ q,
             size_t n, CgWork *w)
{
  double2 s = make_double2(0.0, 0.0);
  for (size_t i = (size_t)blockIdx.x * kCgThreads + threadIdx.x; i < n;
       i += (size_t)gridDim.x * kCgThreads)
  {
    const float2 a = p[i], b = q[i];
    s.x += (double)a.x * b.x + (double)a.y * b.y;
    s.y += (double)a.x * b.y - (double)a.y * b.x;
  }
  grid_sum(s, w, [&](double2 t) {
    const double f = (double)w->rr / (t.x * t.x + t.y * t.y);
    w->a = make_float2((float)(t.x * f), (float)(-t.y * f));
  });
}

// x += a p, r -= a q, beta = ||r_new||^2 / ||r||^2
__global__ void __launch_bounds__(kCgThreads)
    k_cg_update(float2 *__restrict__ x, float2 *__restrict__ r,
                const float2 *__restrict__ p, const float2 *__restrict__ q,
                size_t n, CgWork *w)
{
  const float2 a = w->a;
  double2 s = make_double2(0.0, 0.0);
  for (size_t i = (size_t)blockIdx.x * kCgThreads + threadIdx.x; i < n;
       i += (size_t)gridDim.x * kCgThreads)
  {
    const float2 ap = cmul(a, p[i]), aq = cmul(a, q[i]);
    float2 xv = x[i], rv = r[i];
    xv.x += ap.x;
    xv.y += ap.y;
    rv.x -= aq.x;
    rv.y -= aq.y;
    x[i] = xv;
    r[i] = rv;
    s.x += (double)rv.x * rv.x + (double)rv.y * rv.y;
  }
  grid_sum(s, w, [&](double2 t) {
    const float rr = (float)t.x;
    w->beta = rr / w->rr;
    w->rr = rr;
  });
}

// p = r + beta p
__global__ void __launch_bounds__(kCgThreads)
    k_cg_direction(const float2 *__restrict__ r, float2 *__restrict__ p,
                   size_t n, const CgWork *w)
{
  const float b = w->beta;
  for (size_t i = (size_t)blockIdx.x * kCgThreads + threadIdx.x; i < n;
       i += (size_t)gridDim.x * kCgThreads)
  {
    const float2 rv = r[i];
    float2 pv = p[i];
    pv.x = __fmaf_rn(b, pv.x, rv.x);
    pv.y = __fmaf_rn(b, pv.y, rv.y);
    p[i] = pv;
  }
}

unsigned cg_blocks(size_t n)
{  // four elements a thread until the device is full
  const size_t per = (size_t)kCgThreads * 4;
  return (unsigned)std::min<size_t>(std::max<size_t>((n + per - 1) / per, 1),
                                    kCgMaxBlocks);
}
}  // namespace
}  // namespace gnufft

using namespace gnufft;

extern "C" {

gnufft_status gnufft_cg_begin(const gnufft_plan *plan, const void *residual,
                              uint64_t n, void *work, void *stream)
{
  PlanView v;
  if (!plan_view(plan, &v) || !residual || !work || !n)
    return (gnufft_status)fail(kInvalidArgument, "invalid argument");
  return guarded([&] {
    DeviceGuard dg(v.device);
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    CgWork *w = static_cast<CgWork *>(work);
    GN_CUDA(cudaMemsetAsync(w, 0, offsetof(CgWork, partial), s));
    k_cg_begin<<<cg_blocks(n), kCgThreads, 0, s>>>(
        static_cast<const float2 *>(residual), (size_t)n, w);
    GN_LAUNCH_CHECK("CG start");
  });
}

gnufft_status gnufft_cg_step(const gnufft_plan *plan, void *x, void *residual,
                             void *direction, const void *image, uint64_t n,
                             void *work, void *stream)
{
  PlanView v;
  if (!plan_view(plan, &v) || !x || !residual || !direction || !image ||
      !work || !n)
    return (gnufft_status)fail(kInvalidArgument, "invalid argument");
  return guarded([&] {
    DeviceGuard dg(v.device);
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    CgWork *w = static_cast<CgWork *>(work);
    const unsigned nb = cg_blocks(n);
    float2 *p = static_cast<float2 *>(direction);
    float2 *r = static_cast<float2 *>(residual);
    const float2 *q = static_cast<const float2 *>(image);
    k_cg_dot<<<nb, kCgThreads, 0, s>>>(p, q, (size_t)n, w);
    k_cg_update<<<nb, kCgThreads, 0, s>>>(static_cast<float2 *>(x), r, p, q,
                                          (size_t)n, w);
    k_cg_direction<<<nb, kCgThreads, 0, s>>>(r, p, (size_t)n, w);
    GN_LAUNCH_CHECK("CG step");
  });
}

}  // extern "C"

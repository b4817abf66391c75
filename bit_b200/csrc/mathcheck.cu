// Agreement of the FP64 arithmetic of the near field's pairs with CUDA's exp and rsqrt on the
// device: the largest difference, in units in the last place of CUDA's result, over n seeded
// arguments.  exp: exp_scaled, with and without the check for underflow, kappa log-uniform in [1e-3,
// 1e3] and kappa r uniform in [0, 700) (both with 24 bits, so that their product is exact), and
// exp_tang, t uniform in [-707, 0].  rsqrt: the reciprocal square root inside pair64, both kernels',
// x log-uniform in [1e-12, 1e6].  B200, 16M arguments: exp 1 ulp, rsqrt 2.  A test holds both to a
// bound.
#include "common.cuh"
#include "fp64math.cuh"
#include "near.cuh"
#include "tma.cuh"

namespace bit {

namespace {

// uniform in [0, 1) from a 64-bit mix of the index (splitmix64's finaliser)
__device__ __forceinline__ double unit(unsigned long long i) {
  unsigned long long z = i * 0x9e3779b97f4a7c15ull + 0x632be59bd9b4e019ull;
  z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
  z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
  z ^= z >> 31;
  return (double)(z >> 11) * 0x1p-53;
}

// |a - b| in ulps of b (b finite, non-zero)
__device__ __forceinline__ double ulp_diff(double a, double b) {
  int e;
  frexp(b, &e);
  return fabs(a - b) / ldexp(1.0, e - 53);
}

__global__ void k_math_check(long long n, unsigned long long* worst) {
  __shared__ double2 s_tab[64 * kExpTabCopies];
  exp_tab_fill(s_tab, threadIdx.x, blockDim.x);
  __syncthreads();
  const double2* tab = s_tab + (threadIdx.x & (kExpTabCopies - 1));
  double we = 0.0, wr = 0.0;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    const double t = -707.0 * unit(2 * i);
    const double x = exp10(-12.0 + 18.0 * unit(2 * i + 1));
    we = fmax(we, ulp_diff(exp_tang(t), exp(t)));
    const float kappa = (float)exp10(-3.0 + 6.0 * unit(2 * i + 1));
    const float r = __fdiv_rz((float)(699.9 * unit(2 * i)), kappa);
    const ExpScale k = exp_scale(kappa);
    const double e = exp(-(double)kappa * r);
    we = fmax(we, ulp_diff(exp_scaled<true, kExpTabCopies>(r, k, tab), e));
    we = fmax(we, ulp_diff(exp_scaled<false, kExpTabCopies>(r, k, tab), e));
    // a source of charge 1 at the target, delta = x (kappa = 0: the exponential is 1)
    const double4 one = make_double4(0.0, 0.0, 0.0, 1.0);
    double c = 0.0, s = 0.0;
    pair64<BIT_KERNEL_COULOMB, false, false, false>(0.0, 0.0, 0.0, one, x, k, tab, false, c);
    pair64<BIT_KERNEL_SCREENED, false, false, false>(0.0, 0.0, 0.0, one, x, exp_scale(0.0), tab, false, s);
    wr = fmax(wr, fmax(ulp_diff(c, rsqrt(x)), ulp_diff(s, rsqrt(x))));
  }
  // non-negative doubles order as their bit patterns
  atomicMax(worst, (unsigned long long)__double_as_longlong(we));
  atomicMax(worst + 1, (unsigned long long)__double_as_longlong(wr));
}

// The kernels' give-up path, exercised where no copy is in flight: an mbarrier that no
// copy and no thread ever arrives at, waited on by every thread with the kernels' bounded
// wait (at most `limit` attempts), the outcome combined for the CTA as the near field does,
// and the error flag raised (16) when the wait gives up.
__global__ void k_wait_check(int limit, int* err) {
  __shared__ uint64_t bar;
  if (threadIdx.x == 0) {
    mbar_init(&bar, 1);
    fence_mbar_init();
  }
  __syncthreads();
  const bool landed = mbar_wait(&bar, 0, limit);
  if (__syncthreads_or(!landed) && threadIdx.x == 0) atomicOr(err, 16);
}

// What a near-field queue that gave up may leave: groups with one of their parts done.
__global__ void k_wait_leave(int n, int* part_done) {
  const int g = blockIdx.x * blockDim.x + threadIdx.x;
  if (g < n) part_done[g] = 1;
}

}  // namespace

void device_wait_check(Ctx* c, int limit) {
  for (Tree* t : c->trees)
    if (t->plists.valid) {
      const int n = t->plists.ngroups;
      count_launch(), k_wait_leave<<<grid_for(n, 128), 128, 0, c->stream>>>(n, t->plists.part_done.p);
    }
  count_launch(), k_wait_check<<<1, 128, 0, c->stream>>>(limit, c->dev_err());
  BIT_CHECK_LAUNCH();
  BIT_CUDA(cudaStreamSynchronize(c->stream));
}

void fp64_math_error(Ctx* c, long long n, double* exp_ulps, double* rsqrt_ulps) {
  cudaStream_t s = c->stream;
  DBuf<unsigned long long> w;
  w.ensure(c, 2);
  BIT_CUDA(cudaMemsetAsync(w.p, 0, 2 * sizeof(unsigned long long), s));
  count_launch(), k_math_check<<<c->num_sms * 8, 256, 0, s>>>(n, w.p);
  BIT_CHECK_LAUNCH();
  unsigned long long h[2];
  BIT_CUDA(cudaMemcpyAsync(h, w.p, sizeof(h), cudaMemcpyDeviceToHost, s));
  BIT_CUDA(cudaStreamSynchronize(s));
  *exp_ulps = __builtin_bit_cast(double, h[0]);
  *rsqrt_ulps = __builtin_bit_cast(double, h[1]);
}

}  // namespace bit

// FP64 form of the dynamical core.  Compiled with --fmad=false: every
// multiply and add is rounded separately, exactly as in the FP64
// restatement of the reference, so the two agree bit for bit.
#define ATM_FORM_T double
#define ATM_OPS_NAME ops_fp64
#include "atm_launch.cuh"

namespace atm {

template <bool PK>
static cudaError_t corners_m(const Geom& g, const double* pkap, const double* gz, double* pkapb, double* gzb, int nlev,
                             cudaStream_t s) {
  const StripPlan p = plan_strips(g.nx + 1, g.ny + 1, nlev, COUT, 3, CORN_WARPS_SM);
  return launch(k_corners_m<PK>, p.grid, p.threads, p.threads / MW * CORN_SMEM<PK>, s, g, pkap, gz, pkapb, gzb, p.rows);
}

cudaError_t corners(const Geom& g, const double* pkap, const double* gz, double* pkapb, double* gzb, cudaStream_t s) {
  return corners_m<true>(g, pkap, gz, pkapb, gzb, g.L, s);
}
cudaError_t corners_gz0(const Geom& g, const double* gz, double* gzb, cudaStream_t s) {
  return corners_m<false>(g, nullptr, gz, nullptr, gzb, 1, s);
}

static __global__ void k_pow_log(const double* x, double y, double* p, double* l, int n) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) {
    p[i] = atm_pow(x[i], y);
    l[i] = atm_log(x[i]);
  }
}

// random bit patterns of every exponent, and small integers
__device__ __forceinline__ unsigned long long mix64(unsigned long long z) {
  z += 0x9e3779b97f4a7c15ULL;
  z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ULL;
  z = (z ^ (z >> 27)) * 0x94d049bb133111ebULL;
  return z ^ (z >> 31);
}
static __global__ void k_div_check(unsigned long long n, unsigned long long seed, unsigned long long* bad) {
  unsigned long long local = 0;
  for (unsigned long long i = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; i < n;
       i += (unsigned long long)gridDim.x * blockDim.x) {
    unsigned long long b = mix64(seed * 0x100000001b3ULL + i);
    double x = __longlong_as_double((long long)b);
    if (i % 7 == 0) x = (double)(long long)(b % 2000001) - 1000000.0;
    if (i % 11 == 0) x = __longlong_as_double((long long)(b & 0x800fffffffffffffULL));  // zeros and subnormals
    if (i % 11 == 1) x = __longlong_as_double((long long)(b & 0x8000000000000003ULL));
    if (i % 1000003 == 0) x = copysign(__longlong_as_double(0x7ff0000000000000LL), x);
    bool ok = true;
    double q3 = div_const<3>(x), t3 = x / 3.0;
    double q12 = div_const<12>(x), t12 = x / 12.0;
    ok = ok && (__double_as_longlong(q3) == __double_as_longlong(t3) || (q3 != q3 && t3 != t3));
    ok = ok && (__double_as_longlong(q12) == __double_as_longlong(t12) || (q12 != q12 && t12 != t12));
    double q6 = div_const<6>(x), t6 = x / 6.0;
    ok = ok && (__double_as_longlong(q6) == __double_as_longlong(t6) || (q6 != q6 && t6 != t6));
    const double q = third(x);
    ok = ok && (__double_as_longlong(q) == __double_as_longlong(t3) || (q != q && t3 != t3));
    if (!ok) ++local;
  }
  if (local) atomicAdd(bad, local);
}

cudaError_t device_div_check(unsigned long long n, unsigned long long seed, unsigned long long* bad, cudaStream_t s) {
  k_div_check<<<1184, 256, 0, s>>>(n, seed, bad);
  return cudaGetLastError();
}

// A bounded mbarrier wait, made to run out: one thread arms an mbarrier for 16
// bytes of transactions that no copy ever brings (no copy is issued) and waits
// on it with a poll limit; it must come back with the failure recorded in
// *flag.
__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}

__device__ __forceinline__ void fence_mbar_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
               : "memory");
}

// wait for a phase of the barrier, at most max_iter polls of at most ~1 us
// each; true on success
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t phase, int max_iter) {
  uint32_t done = 0;
  for (int it = 0; it < max_iter; ++it) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, 1000;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(smem_u32(bar)), "r"(phase)
        : "memory");
    if (done) return true;
  }
  return false;
}

static __global__ void k_wait_timeout(int max_polls, int* flag) {
  __shared__ __align__(8) uint64_t bar;
  if (threadIdx.x == 0) {
    mbar_init(&bar, 1);
    fence_mbar_init();
    mbar_expect_tx(&bar, 16);
    const bool ok = mbar_wait(&bar, 0, max_polls);
    *flag = ok ? 0 : 1;
  }
}

cudaError_t device_wait_timeout(int max_polls, int* flag, cudaStream_t s) {
  k_wait_timeout<<<1, 32, 0, s>>>(max_polls, flag);
  return cudaGetLastError();
}

cudaError_t device_pow_log(const double* x, double y, double* p, double* l, int n, cudaStream_t s) {
  k_pow_log<<<(n + 255) / 256, 256, 0, s>>>(x, y, p, l, n);
  return cudaGetLastError();
}

}  // namespace atm

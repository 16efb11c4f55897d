"""The samplers' divisions and logarithm (common.cuh, stoch_device.cuh) against the operator and
the general logarithm, compiled as the run-time kernels are: every argument of a draw's
logarithm, every significand of a divisor, the waiting times of hazards of every
significand, the search's quotients, and the Poisson counts near their decision."""
import pytest

from nvrtc_kernels import Kernels

pytestmark = pytest.mark.gpu

SRC = r'''#include "stoch_device.cuh"
using namespace gpgmp;
__device__ __forceinline__ unsigned mix(unsigned x) {
  x ^= x >> 16; x *= 0x7feb352du; x ^= x >> 15; x *= 0x846ca68bu; return x ^ (x >> 16);
}
__device__ __forceinline__ bool same(float a, float b) { return __float_as_uint(a) == __float_as_uint(b); }
// 2^24 threads
extern "C" __global__ void check_log(unsigned* bad) {
  const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
  const float a = log_draw(i << 8 | (mix(i) & 255u)), b = gp_logf(u01_open0(i << 8));
  if (!(a == b)) atomicAdd(bad, 1u);
}
// 2^23 threads: divisors of every significand at three exponents, dividends at random and powers of two
extern "C" __global__ void check_wait(unsigned* bad) {
  const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
  const unsigned exps[3] = {127u - 59u, 127u, 127u + 59u};
  for (int e = 0; e < 3; ++e) {
    const float h0 = __uint_as_float(exps[e] << 23 | i);
    for (int k = 0; k < 24; ++k) {
      const unsigned v = k < 8 ? 0xffffffu - k : k < 16 ? (1u << 24) - (1u << k) : mix(24u * i + k) >> 8;
      const unsigned w = (v - 1u) << 8;
      if (!(ssa_wait(w, h0) == -gp_logf(u01_open0(w)) / h0)) atomicAdd(bad, 1u);
    }
  }
}
// 2^23 threads: div_mid's reciprocal, and its quotients of powers of two and random dividends
extern "C" __global__ void check_recip(unsigned* bad) {
  const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
  const unsigned exps[4] = {127u - 59u, 127u, 128u, 127u + 59u};
  for (int e = 0; e < 4; ++e) {
    const float b = __uint_as_float(exps[e] << 23 | i);
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(b));
    y = fmaf(fmaf(-b, y, 1.0f), y, y);
    if (!same(y, 1.0f / b)) atomicAdd(bad, 1u);
    for (int k = 0; k < 16; ++k) {
      const float a = __uint_as_float((127u - 8u + k) << 23 | (k & 1 ? mix(16u * i + k) & 0x7fffffu : 0u));
      if (!same(div_mid(a, b), a / b)) atomicAdd(bad, 1u);
    }
  }
}
// 2^23 threads: the search's terms over its constant and table divisors
extern "C" __global__ void check_small(unsigned* bad) {
  const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
  const unsigned exps[2] = {127u, 127u - 90u};
  for (int e = 0; e < 2; ++e)
    for (int k = 0; k < kRecipMax; ++k) {
      const float a = __uint_as_float(exps[e] << 23 | i), b = (float)(k + 1);
      if (!same(div_small(a, b, kRecip[k]), a / b)) atomicAdd(bad, 1u);
    }
}
// counts with the mean on, just below and just above an arrival's time
extern "C" __global__ void check_poisson(unsigned* bad, int n) {
  const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (unsigned)n) return;
  const float tops[4] = {1.0f, 30.0f, 250.0f, 300.0f};
  Stream from; from.init(7u, i, 1u, 2u, 3u);
  for (int q = 0; q < 4; ++q) {
    Stream st = from;
    float t = 0.0f;
    const float top = tops[q] * u01(mix(i + q));
    while (t <= top) t = t - log_draw(st.next());
    for (int d = -3; d <= 3; ++d) {
      const float lam = __uint_as_float(__float_as_uint(t) + d);
      Stream a = from, b = from;
      if (poisson(a, lam) != poisson_exact(b, lam)) atomicAdd(bad, 1u);
    }
  }
  const float edge[4] = {255.99998f, 256.0f, 1e-30f, 0.0f};
  for (int q = 0; q < 4; ++q) {
    Stream a = from, b = from;
    if (poisson(a, edge[q]) != (edge[q] > 0.0f ? poisson_exact(b, edge[q]) : 0)) atomicAdd(bad, 1u);
  }
}
'''


@pytest.fixture(scope="module")
def kernels():
    k = Kernels(SRC)
    yield k
    k.close()


@pytest.mark.parametrize("name,threads,ints", [("check_log", 1 << 24, ()), ("check_wait", 1 << 23, ()),
                                               ("check_recip", 1 << 23, ()),
                                               ("check_small", 1 << 23, ()), ("check_poisson", 1 << 15, (1 << 15,))])
def test_rounding(gpgmp, kernels, name, threads, ints):
    import torch
    bad = torch.zeros(1, dtype=torch.int32, device="cuda")
    kernels.launch(name, threads // 256, 256, bad, *ints)
    torch.cuda.synchronize()
    assert int(bad.item()) == 0

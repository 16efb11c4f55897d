"""A long scan beside a kernel that holds an SM: the scan runs on the others."""
import time

import pytest

from nvrtc_kernels import Kernels

pytestmark = pytest.mark.gpu

# one block that takes an SM's shared memory for `ms` milliseconds (and stops by itself after
# 2^28 polls)
SRC = r'''
extern "C" __global__ void hold(unsigned* out, int ms) {
  extern __shared__ unsigned s[];
  unsigned long long t0, t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t0));
  s[threadIdx.x] = 1u;
  for (unsigned i = 0; i < (1u << 28); ++i) {
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    if (t - t0 > 1000000ull * (unsigned)ms) break;
  }
  out[threadIdx.x] = s[threadIdx.x];
}
'''


def test_scan_on_the_free_sms(gpgmp):
    import torch
    from inchman_b200 import individual as ind
    n = 300 * 16384 + 77
    x = torch.randint(0, 1 << 20, (n,), device="cuda", dtype=torch.int32)
    scratch = ind.scan_scratch(n)
    want = ind.exclusive_scan_u32(x, scratch)
    k = Kernels(SRC)
    out = torch.zeros(32, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    held, done = torch.cuda.Event(), torch.cuda.Event()
    k.launch("hold", 1, 32, out, 300, smem=220 * 1024, stream=a)
    held.record(a)
    time.sleep(0.02)
    with torch.cuda.stream(b):
        got = ind.exclusive_scan_u32(x, scratch)
        done.record(b)
    done.synchronize()
    finished_first = not held.query()
    torch.cuda.synchronize()
    k.close()
    assert torch.equal(got, want) and int(out.sum()) == 32
    assert finished_first and ind.scratch_status(scratch, 0) == 0

"""Operands that the kernel directly in front of a linear has written.  The linear's kernels start before that kernel is done
(programmatic dependent launch) and may read ahead of their wait nothing that it writes: the results are those of the same
calls with the device idle in between."""
import pytest
import torch

import xla_b200
from tests import qmm_cases as qc

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("scale_dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("variant,wbits,bs,zp,N,K,M", [
    ("i8mma", 4, 128, True, 8192, 2048, 3), ("i8mma", 8, 64, False, 4096, 2048, 2), ("i8mma", 4, 64, True, 4096, 2048, 1),
    ("mma", 4, 128, False, 8192, 2048, 16), ("mma", 8, 128, False, 8192, 2048, 32), ("mma", 4, 256, False, 8192, 2048, 5),
    ("tmem", 4, 128, True, 8192, 2048, 29), ("tmem", 8, -1, True, 4096, 2048, 200), ("i8tc", 4, 128, True, 8192, 2048, 40),
    ("i8tc", 4, 128, False, 8192, 2048, 16), ("i8tc", 8, -1, False, 4096, 2048, 300),
])
def test_operands_written_by_the_kernel_in_front(scale_dtype, variant, wbits, bs, zp, N, K, M):
  g = qc.gen(N + K + M)
  w = (qc.int4_weight if wbits == 4 else qc.int8_weight)(g, N, K).to(DEV)
  wk = xla_b200.pack_int4(w) if wbits == 4 else w
  x0 = qc.activations(g, M, K).to(DEV)
  s0 = (qc.per_channel_scale(g, N) if bs == -1 else qc.blockwise_scale(g, K // bs, N)).to(scale_dtype).to(DEV)
  z0 = (3 * s0) if zp else None
  x, s, z = x0.clone(), s0.clone(), None if z0 is None else z0.clone()

  def linear():
    return torch.ops.xla_b200.quantized_matmul_packed(x, wk, s, z, block_size=bs, int4_weight=wbits == 4, weight_is_packed=wbits == 4,
                                                      out_dtype=torch.float32)

  def calls(idle):
    outs = []
    for i in range(12):
      factor = 2.0**(i % 5 - 2)
      for target, origin in ((s, s0), (x, x0), (z, z0))[i % 3:] + ((s, s0), (x, x0), (z, z0))[:i % 3]:
        if origin is not None:
          torch.mul(origin, factor, out=target)
          if idle:
            torch.cuda.synchronize()
      outs.append(linear())
      if idle:
        torch.cuda.synchronize()
    return outs

  with xla_b200.force_variant(variant):
    want = calls(True)
    for _ in range(3):
      for a, b in zip(calls(False), want):
        assert torch.equal(a, b)


@pytest.mark.parametrize("M", [1, 16, 80])
def test_weights_packed_directly_in_front(M):
  g = qc.gen(M)
  N, K, bs = 4096, 2048, 128
  x, s = qc.activations(g, M, K).to(DEV), qc.blockwise_scale(g, K // bs, N).to(DEV)
  ws = [qc.int4_weight(g, N, K).to(DEV) for _ in range(4)]

  def run(w, idle):
    mod = xla_b200.XlaQuantizedLinear(K, N, is_symmetric=True, block_size=bs, int4_weight=True)
    mod.load_quantized_weight(qc.to_sbn(w, bs), s)
    if idle:
      mod._packed_weight()
      torch.cuda.synchronize()
    return mod(x)

  want = [run(w, True) for w in ws]
  torch.cuda.synchronize()
  got = [run(w, False) for w in ws]
  assert all(torch.equal(a, b) for a, b in zip(got, want))


def test_two_streams_at_once():
  """Launches whose CTAs wait for one another's partial sums, on two streams that share the SMs: nobody waits for a CTA that
  has not started."""
  from xla_b200 import _capi
  assert _capi.device_error(DEV) == 0
  g = qc.gen(3)
  cases = []
  for variant, wbits, bs, N, K, M in (("tmem", 4, 128, 2560, 8192, 29), ("i8tc", 4, 128, 5120, 8192, 40), ("i8tc", 8, -1, 2560, 8192, 16)):
    w = (qc.int4_weight if wbits == 4 else qc.int8_weight)(g, N, K).to(DEV)
    s = (qc.per_channel_scale(g, N) if bs == -1 else qc.blockwise_scale(g, K // bs, N)).to(DEV)
    cases.append((variant, qc.activations(g, M, K).to(DEV), xla_b200.pack_int4(w) if wbits == 4 else w, s, bs, wbits == 4))

  def run(c):
    variant, x, w, s, bs, int4 = c
    with xla_b200.force_variant(variant):
      return torch.ops.xla_b200.quantized_matmul_packed(x, w, s, block_size=bs, int4_weight=int4, weight_is_packed=int4,
                                                        out_dtype=torch.float32)

  want = [run(c) for c in cases]
  torch.cuda.synchronize()
  streams = [torch.cuda.Stream(), torch.cuda.Stream()]
  outs = []
  for i in range(60):
    for j, st in enumerate(streams):
      with torch.cuda.stream(st):
        outs.append(((i + j) % 3, run(cases[(i + j) % 3])))
  torch.cuda.synchronize()
  assert _capi.device_error(DEV) == 0
  assert all(torch.equal(y, want[k]) for k, y in outs)

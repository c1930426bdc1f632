"""A module's scales and zero points are read on every call, in the type they are held in: 16-bit ones give the bits of the
fp32 call with the same values in every kernel that a module reaches, and a write to the buffers shows in the next call
however it was made.  (Scale blocks in a buffer at an odd element, and in the tensor-memory kernel an odd number of them, are converted first.)"""
import pytest
import torch

import xla_b200
from tests import qmm_cases as qc

pytestmark = pytest.mark.gpu
DEV = "cuda:0"

# weight bits, block size, zero points, activation quantization, N, K, M, whether the buffers start at an odd element
CASES = [
    (8, -1, False, False, 261, 1056, 1, True), (8, -1, True, False, 512, 1024, 2, False), (4, 128, False, False, 1024, 4096, 1, False),
    (4, 128, True, False, 1024, 4096, 3, False), (4, 64, True, False, 130, 320, 2, False), (8, 128, False, False, 4096, 512, 2, False),
    (4, 128, False, False, 1024, 2048, 8, False), (8, -1, False, False, 512, 1024, 14, False), (8, 256, False, False, 514, 1024, 29, True),
    (4, 128, True, False, 4096, 1024, 29, False), (4, -1, True, False, 777, 4096, 130, True), (4, 64, False, False, 300, 1024, 40, False),
    (8, 128, False, False, 1000, 2048, 70, False), (8, -1, False, False, 1025, 2048, 300, True), (8, 256, True, False, 2048, 1024, 9, False),
    (4, 256, False, False, 4096, 2048, 520, False), (8, -1, False, True, 514, 1024, 4, False), (8, -1, True, True, 300, 1024, 40, True),
    (8, -1, True, True, 300, 512, 10, False), (4, 128, True, False, 301, 1024, 29, False), (8, 64, True, False, 300, 832, 9, True),
    # odd row counts: 16-bit pairs that span two blocks; with an odd number of blocks a last value that has no partner
    (4, 128, False, False, 1027, 128 * 33, 1, False), (8, 64, True, False, 33, 192, 2, False), (4, 64, True, False, 131, 320, 5, False),
    (4, 128, True, False, 257, 128 * 9, 40, False), (8, 64, True, False, 385, 64 * 15, 33, False), (4, 128, False, False, 129, 128 * 31, 16, False),
    (4, 128, False, False, 4097, 128 * 63, 24, False), (4, 256, False, False, 3841, 256 * 17, 12, False), (8, 128, False, False, 513, 128 * 21, 100, False),
    (4, 128, True, False, 1023, 128 * 17, 16, False), (4, 128, True, False, 1023, 128 * 16, 29, False),
    (4, 128, True, False, 257, 128 * 10, 3, False), (4, 64, True, False, 131, 384, 5, False), (4, 128, False, False, 4097, 128 * 64, 24, False),
    (8, 64, True, False, 385, 64 * 16, 33, False), (4, 256, False, False, 3841, 256 * 16, 12, False),
    # shapes that only the any-shape and the GEMV kernel take, which read fp32 scales
    (8, -1, True, False, 40, 72, 5, False), (8, -1, True, False, 40, 48, 5, True), (8, 4, False, False, 12, 20, 3, False),
    (8, -1, True, True, 40, 72, 5, False),
    # small weights above 32 tokens: the conversion kernel
    (4, -1, False, False, 1976, 1504, 45, True), (8, -1, False, False, 269, 1536, 300, False), (8, 128, False, False, 301, 1024, 45, True),
]


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("wbits,bs,zp,qact,N,K,M,odd", CASES)
def test_module_follows_its_scales(dtype, wbits, bs, zp, qact, N, K, M, odd):
  g = qc.gen(N + K + M)
  x = qc.activations(g, M, K, dtype).to(DEV)
  w = (qc.int4_weight if wbits == 4 else qc.int8_weight)(g, N, K)
  native = xla_b200.pack_int4(w.to(DEV)) if wbits == 4 and K % 2 == 0 and not qact else w.to(DEV)

  def held(t):
    flat = torch.empty(t.numel() + 1, dtype=dtype, device=DEV)[1 if odd else 0:][:t.numel()]
    return flat.copy_(t.flatten()).view(t.shape)

  def draw():
    s = qc.per_channel_scale(g, N) if bs == -1 else qc.blockwise_scale(g, K // bs, N)
    return s.to(dtype), (torch.randint(-3, 4, s.shape, generator=g) * s).to(dtype) if zp else None

  def in_f32(s, z):
    return torch.ops.xla_b200.quantized_matmul_packed(x, native, s.float().to(DEV), None if z is None else z.float().to(DEV),
                                                      block_size=bs, int4_weight=wbits == 4, weight_is_packed=native.dtype == torch.uint8,
                                                      quantize_activation=qact, out_dtype=dtype)

  mod = xla_b200.XlaQuantizedLinear(K, N, is_symmetric=not zp, block_size=bs, int4_weight=wbits == 4, quantize_activation=qact)
  s, z = draw()
  mod.load_quantized_weight((w if bs == -1 else qc.to_sbn(w, bs)).to(DEV), held(s), None if z is None else held(z))
  assert torch.equal(mod(x), in_f32(s, z))
  s, z = draw()
  mod.weight_scaler.data.copy_(s)  # leaves the version counter as it is, as a replayed graph does
  if z is not None:
    mod.zero_point.data.copy_(z)
  y = mod(x)
  assert y.dtype == dtype and torch.equal(y, in_f32(s, z))


@pytest.mark.parametrize("wbits,bs", [(4, 128), (4, -1), (8, 128), (8, -1)])
def test_module_follows_its_weight(wbits, bs):
  """The K-minor weight that a module keeps is made again when the buffer is written in place or replaced; other scales in
  another type need nothing."""
  g = qc.gen(11)
  N, K, M = 256, 1024, 3
  x = qc.activations(g, M, K).to(DEV)
  layout = lambda w: (w if bs == -1 else qc.to_sbn(w, bs)).to(DEV)  # noqa: E731
  weights = [(qc.int4_weight if wbits == 4 else qc.int8_weight)(g, N, K) for _ in range(3)]
  s = (qc.per_channel_scale(g, N) if bs == -1 else qc.blockwise_scale(g, K // bs, N)).to(DEV)

  def fresh(w, scale):
    m = xla_b200.XlaQuantizedLinear(K, N, is_symmetric=True, block_size=bs, int4_weight=wbits == 4)
    m.load_quantized_weight(layout(w), scale)
    return m

  mod = fresh(weights[0], s)
  assert torch.equal(mod(x), fresh(weights[0], s)(x))
  mod.weight.copy_(layout(weights[1]))
  assert torch.equal(mod(x), fresh(weights[1], s)(x))
  mod.weight = layout(weights[2])
  assert torch.equal(mod(x), fresh(weights[2], s)(x))
  mod.weight_scaler = s.bfloat16()
  y = mod(x)
  assert y.dtype == torch.bfloat16 and torch.equal(y, fresh(weights[2], s.bfloat16())(x))

"""The GEMM on pairs of CTAs where its tiling can go wrong, against the any-shape kernel or in 64 bits: ragged rows
(a second CTA without any), a token more or less than a tile, K that ends inside a stage, more tiles than pairs, split items."""
import pytest
import torch

import xla_b200
from oracle import qmm_oracle as qo
from tests import qmm_cases as qc

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("M,N,K,zp", [
    (16, 300, 512, False), (33, 1031, 80, False), (255, 2050, 144, True), (256, 1026, 4096, False), (257, 1026, 1040, True),
    (520, 129, 2064, False), (64, 4096, 4096, True), (2300, 2304, 1152, False),
])
def test_w8a8_is_exact(M, N, K, zp, dtype):
  """Whole-number sums and the reference's order of the products behind them: every bit, also in rows that TMA could not store."""
  g = qc.gen(M + N + K)
  x, w, s = qc.activations(g, M, K, dtype), qc.int8_weight(g, N, K), qc.per_channel_scale(g, N)
  z = torch.randint(-20, 21, (N,), generator=g) * s if zp else None
  args = x.to(DEV), w.to(DEV), s.to(DEV), None if z is None else z.to(DEV)
  with xla_b200.force_variant("generic"):
    ref = torch.ops.xla.quantized_matmul(*args, quantize_activation=True)
  assert torch.equal(torch.ops.xla.quantized_matmul(*args, quantize_activation=True), ref)


@pytest.mark.parametrize("x_dt,out_dt", [(torch.bfloat16, torch.bfloat16), (torch.float16, torch.float16), (torch.bfloat16, torch.float32),
                                         (torch.float32, torch.float32)])
@pytest.mark.parametrize("M,N,K,zp", [
    (128, 10241, 256, False), (129, 9986, 400, False), (84, 10240, 272, True), (85, 10242, 272, True), (333, 2560, 1168, True),
    (300, 19200, 640, False), (100, 4098, 8208, False), (100, 4096, 8208, True), (1100, 2600, 512, False),
])
def test_weight_only(M, N, K, zp, x_dt, out_dt):
  g = qc.gen(M + N + K)
  x = qc.activations(g, M, K, x_dt, outliers=True).to(DEV)
  w, s = qc.int8_weight(g, N, K).to(DEV), qc.per_channel_scale(g, N).to(DEV)
  z = (torch.randint(-20, 21, (N,), generator=g).to(DEV) * s) if zp else None
  with xla_b200.force_variant("i8tc"):
    run = lambda: torch.ops.xla_b200.quantized_matmul_packed(x, w, s, z, out_dtype=out_dt)  # noqa: E731
    out = run()
    assert all(torch.equal(out, run()) for _ in range(3))
  exact = (x.double() @ w.double().T) * s.double()
  if zp:
    exact -= x.double().sum(1, keepdim=True) * z.double()
  # three limbs: 2^-22 of the row's largest value per activation; two (16-bit results without zero points): 2^-15 of it, under
  # the rounding of the result
  assert qo.max_abs_rel(out, exact) < {torch.float32: 1e-5, torch.float16: 3e-3, torch.bfloat16: 1e-2}[out_dt]


@pytest.mark.parametrize("M,N,K,zp", [(129, 11008, 384, False), (256, 11008, 384, False), (100, 4096, 12288, False), (92, 5120, 640, True), (128, 5120, 640, True),
                                       (129, 3584, 12288, False), (129, 3840, 12288, True), (129, 9500, 12288, False)])
def test_both_sides_of_the_line_between_pairs_and_single_ctas(M, N, K, zp):
  """A round of tiles less on pairs than on single CTAs, and the same number; K long enough to be split."""
  g = torch.Generator(device=DEV).manual_seed(M + N + K)
  x = torch.randn(M, K, generator=g, device=DEV).bfloat16()
  w = torch.randint(-127, 128, (N, K), generator=g, device=DEV, dtype=torch.int8)
  s = (torch.rand(N, generator=g, device=DEV) + 0.5) / 73 / K**0.5
  z = torch.randint(-20, 21, (N,), generator=g, device=DEV) * s if zp else None
  with xla_b200.force_variant("i8tc"):
    out = torch.ops.xla_b200.quantized_matmul_packed(x, w, s, z, out_dtype=torch.float32)
  exact = (x.double() @ w.double().T) * s.double() - (x.double().sum(1, keepdim=True) * z.double() if zp else 0.)
  assert qo.max_abs_rel(out, exact) < 1e-5  # three limbs: 2^-22 of the row's largest value per activation

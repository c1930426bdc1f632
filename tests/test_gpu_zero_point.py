"""Zero points inside the tensor-core kernels against the CPU oracle: one and several token tiles, K split over CTAs, scale
blocks of both kinds, chunked batches, fp32 activations."""
import pytest
import torch

import xla_b200
from oracle import qmm_oracle as qo
from tests import qmm_cases as qc

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("wbits,bs,N,K,M,dtype", [
    (8, -1, 300, 1056, 17, torch.bfloat16), (8, 128, 1000, 1280, 33, torch.float16), (8, 256, 129, 768, 70, torch.bfloat16),
    (4, 128, 4096, 2048, 29, torch.float16), (4, 128, 777, 1024, 64, torch.bfloat16), (4, -1, 520, 4096, 130, torch.bfloat16),
    (4, 256, 300, 1024, 513, torch.float16), (8, -1, 260, 272, 1100, torch.float32), (4, 128, 4096, 1024, 40, torch.float32),
    (8, 512, 200, 1024, 9, torch.float32), (8, 64, 300, 832, 40, torch.float32), (4, 64, 520, 1088, 9, torch.float32),
  (4, 64, 300, 4096, 200, torch.float32),
])
def test_zero_points_above_eight_tokens(wbits, bs, N, K, M, dtype):
  g = qc.gen(N + K + M)
  x = qc.activations(g, M, K, dtype, outliers=True)
  w = qc.int4_weight(g, N, K) if wbits == 4 else qc.int8_weight(g, N, K)
  s = qc.per_channel_scale(g, N) if bs == -1 else qc.blockwise_scale(g, K // bs, N)
  zp = torch.randint(-3, 4, s.shape, generator=g).float() * s
  exact = qo.quantized_matmul(x.float(), w if bs == -1 else qc.to_sbn(w, bs), s, zp, block_size=bs, dot_round=None)
  wd = xla_b200.pack_int4(w.to(DEV)) if wbits == 4 else w.to(DEV)
  for out_dtype, tol in ((torch.float32, 1e-5), (torch.bfloat16, 1e-2)):
    out = torch.ops.xla_b200.quantized_matmul_packed(x.to(DEV), wd, s.to(DEV), zp.to(DEV), block_size=bs, int4_weight=wbits == 4,
                                                     weight_is_packed=wbits == 4, out_dtype=out_dtype)
    assert qo.max_abs_rel(out, exact) < tol, out_dtype


@pytest.mark.parametrize("variant", ["auto", "tmem"])
@pytest.mark.parametrize("M", [9, 32, 70])
@pytest.mark.parametrize("wbits,K", [(8, k) for k in (64, 80, 96, 112, 128, 144, 160, 176, 192, 208, 224, 240, 256, 272)] +
                         [(4, k) for k in (64, 96, 128, 160, 192, 224, 256, 288)])
def test_zero_points_per_channel_on_few_inputs(wbits, K, M, variant):
  """The sum over all of a row, from eight lanes' worth of values to more than a warp's.  AUTO on both sides of its lines (1030
  outputs, and enough items for the tensor-memory kernel above 64 tokens)."""
  for N in ((1030, 12290) if variant == "auto" else (130,)):
    g = qc.gen(N + K + M)
    x = (torch.rand(M, K, generator=g) + 0.5).bfloat16().to(DEV)  # a sum in which a value left out shows
    w = (qc.int4_weight if wbits == 4 else qc.int8_weight)(g, N, K).to(DEV)
    s = qc.per_channel_scale(g, N).to(DEV)
    z = torch.randint(-20, 21, (N,), generator=g).to(DEV) * s
    with xla_b200.force_variant(variant):
      out = torch.ops.xla_b200.quantized_matmul_packed(x, xla_b200.pack_int4(w) if wbits == 4 else w, s, z, int4_weight=wbits == 4,
                                                       weight_is_packed=wbits == 4, out_dtype=torch.float32)
    exact = (x.double() @ w.double().T) * s.double() - x.double().sum(1, keepdim=True) * z.double()
    # exact products (or 2^-22 of the row's largest activation); K additions in fp32 at most: K 2^-24 < 2e-5 of the largest result
    assert qo.max_abs_rel(out, exact) < 2e-5


@pytest.mark.parametrize("wbits,bs,K,M", [(8, -1, 2032, 20), (8, -1, 2048, 20), (8, -1, 2064, 9), (4, -1, 4128, 70), (8, -1, 12304, 33),
                                          (4, 384, 7680, 300), (8, 256, 4096, 513), (4, 2048, 8192, 40)])
def test_sums_of_long_rows_and_many_blocks(wbits, bs, K, M):
  """A row per warp and per CTA, on both sides of the line; more pieces than a few CTAs have warps."""
  g = qc.gen(K + M)
  N = 130
  x = (torch.rand(M, K, generator=g) + 0.5).bfloat16().to(DEV)
  w = (qc.int4_weight if wbits == 4 else qc.int8_weight)(g, N, K).to(DEV)
  s = (qc.per_channel_scale(g, N) if bs == -1 else qc.blockwise_scale(g, K // bs, N)).to(DEV)
  z = torch.randint(-20, 21, s.shape, generator=g).to(DEV) * s
  with xla_b200.force_variant("tmem"):
    out = torch.ops.xla_b200.quantized_matmul_packed(x, xla_b200.pack_int4(w) if wbits == 4 else w, s, z, block_size=bs,
                                                     int4_weight=wbits == 4, weight_is_packed=wbits == 4, out_dtype=torch.float32)
  S = 1 if bs == -1 else K // bs
  xb, wb = x.double().view(M, S, -1), w.double().view(N, S, -1)
  exact = torch.einsum("msk,nsk,sn->mn", xb, wb, s.double().view(S, N)) - torch.einsum("ms,sn->mn", xb.sum(-1), z.double().view(S, N))
  # the sums of positive activations: a lane adds K / 32 of them at most in fp32, the products' sums fewer in a row
  assert qo.max_abs_rel(out, exact) < 2e-5

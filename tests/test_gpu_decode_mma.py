"""The conversions of `decode_mma.cu`: every int4 and int8 value, for each number of warps per tile and both token ranges of the kernel."""
import pytest
import torch

import xla_b200
from tests import qmm_cases as qc

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("wbits,bs,N", [(4, 128, 16 * 896), (4, 256, 16 * 897 - 8), (4, -1, 16 * 896), (4, 128, 4096), (8, 128, 16 * 1792), (8, -1, 2048)])
@pytest.mark.parametrize("M", [1, 4, 5, 8, 9, 32])
def test_every_weight_value_is_converted_exactly(dtype, wbits, bs, N, M):
  """Small whole activations and scales of one: the fp32 result is a whole number, equal to the integer product.  Four warps per
  tile (int4 from 896 row tiles on) convert in one way up to four tokens and in another from five."""
  K = 1024 + 512 * (M % 2)
  g = qc.gen(N + M)
  lo, hi = (-8, 8) if wbits == 4 else (-128, 128)
  w = (torch.arange(N * K, dtype=torch.int32).reshape(N, K) * 7 % (hi - lo) + lo).to(torch.int8).to(DEV)
  x = torch.randint(-2, 3, (M, K), generator=g).to(DEV)
  s = torch.ones((N,) if bs == -1 else (K // bs, N), device=DEV)
  wd = xla_b200.pack_int4(w) if wbits == 4 else w
  with xla_b200.force_variant("mma"):
    out = torch.ops.xla_b200.quantized_matmul_packed(x.to(dtype), wd, s, block_size=bs, int4_weight=wbits == 4,
                                                     weight_is_packed=wbits == 4, out_dtype=torch.float32)
  assert torch.equal(out.double(), x.double() @ w.double().T)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("M", [1, 5, 8])
@pytest.mark.parametrize("bs,N,K", [(128, 2368, 2048), (128, 2368, 2176), (-1, 2369, 2176), (-1, 257, 4096), (384, 2000, 4992), (128, 16, 4224), (-1, 512, 512), (128, 1447, 1792)])
def test_few_row_tiles(dtype, bs, N, K, M):
  """int4 with a row tile per SM at most (2368 rows on 148) takes its activations a step ahead from 17 steps on: whole numbers again."""
  g = qc.gen(N + K + M)
  w = (torch.arange(N * K, dtype=torch.int32).reshape(N, K) * 7 % 16 - 8).to(torch.int8).to(DEV)
  x = torch.randint(-2, 3, (M, K), generator=g).to(DEV)
  s = torch.ones((N,) if bs == -1 else (K // bs, N), device=DEV)
  with xla_b200.force_variant("mma"):
    out = torch.ops.xla_b200.quantized_matmul_packed(x.to(dtype), xla_b200.pack_int4(w), s, block_size=bs, int4_weight=True,
                                                     weight_is_packed=True, out_dtype=torch.float32)
  assert torch.equal(out.double(), x.double() @ w.double().T)

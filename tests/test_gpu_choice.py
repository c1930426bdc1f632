"""AUTO's choice of kernel on both sides of its lines, by name (16-bit results), with a result against 64 bits."""
import pytest
import torch

import xla_b200
from oracle import qmm_oracle as qo
from xla_b200 import _capi

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def chosen(wbits, bs, zp, M, N, K):
  return _capi.lib().qmm_weight_only_variant_for(wbits, M, N, K, max(bs, 0), int(zp)).decode()


def call_and_exact(wbits, bs, zp, M, N, K, out_dtype, dtype=torch.bfloat16):
  g = torch.Generator(device=DEV).manual_seed(M + N + K)
  x = torch.randn(M, K, generator=g, device=DEV)
  x = torch.where(torch.rand(M, K, generator=g, device=DEV) < 0.01, x * 20, x).to(dtype)
  lo, hi = (-8, 8) if wbits == 4 else (-127, 128)
  w = torch.randint(lo, hi, (N, K), generator=g, device=DEV, dtype=torch.int8)
  S = 1 if bs == -1 else K // bs
  s = (torch.rand((N,) if bs == -1 else (S, N), generator=g, device=DEV) + 0.5) / (4.6 if wbits == 4 else 73) / K**0.5
  z = torch.randint(-2, 3, s.shape, generator=g, device=DEV) * s if zp else None
  wd = xla_b200.pack_int4(w) if wbits == 4 else w
  call = lambda: torch.ops.xla_b200.quantized_matmul_packed(x, wd, s, z, block_size=bs, int4_weight=wbits == 4,  # noqa: E731
                                                            weight_is_packed=wbits == 4, out_dtype=out_dtype)
  xb = x.double().view(M, S, -1)
  exact = torch.einsum("msk,nsk,sn->mn", xb, w.double().view(N, S, -1), s.double().view(S, N))
  if zp:
    exact -= torch.einsum("ms,sn->mn", xb.sum(-1), z.double().view(S, N))
  return call, exact


@pytest.mark.parametrize("wbits,bs,zp,M,N,K,kernel", [
    (4, 64, False, 33, 512, 960, "tmem"), (8, 64, False, 64, 512, 960, "tmem"), (4, 64, False, 65, 512, 960, "tcgen05"),
    (8, 64, False, 576, 512, 19968, "tcgen05"), (8, 64, False, 576, 512, 20032, "tmem"), (4, 64, False, 1152, 512, 8000, "tcgen05"),
    (4, 64, False, 1152, 512, 8064, "tmem"), (8, 64, False, 1143, 1024, 3392, "tcgen05"), (8, 64, False, 1143, 1024, 3456, "tmem"),
    (4, 64, False, 256, 1024, 9984, "tcgen05"), (4, 64, False, 256, 1024, 10048, "tmem"),
    (8, 64, False, 1217, 1024, 1344, "tmem"), (8, 64, False, 8, 8192, 7424, "mma"), (8, 64, False, 9, 8192, 4160, "tmem"),
    (8, 128, False, 1100, 1024, 1152, "tmem"), (8, 256, False, 1100, 260, 1024, "tmem"), (8, 128, False, 1024, 1024, 1152, "i8tc"),
    (8, -1, False, 1100, 1024, 1040, "tmem"),
    # int4 blocks of few tokens: from 80 million values, more weight tiles than SMs (18944 outputs), long blocks, and blocks that i8tc leaves
    (4, 128, False, 9, 11008, 8192, "i8tc"), (4, 128, False, 10, 8448, 8192, "tmem"), (4, 128, False, 11, 11008, 8192, "tmem"),
    (4, 128, False, 10, 18945, 3584, "i8tc"), (4, 128, False, 10, 18944, 3584, "tmem"), (4, 256, False, 16, 22016, 3584, "i8tc"),
    (4, 128, False, 16, 22016, 3584, "tmem"), (4, 256, False, 17, 22016, 3584, "tmem"), (4, 64, False, 9, 33024, 4160, "tmem"),
    # zero points at two to eight tokens: blocks of 64, more weight tiles than SMs
    (4, 64, True, 8, 14336, 4096, "i8mma"), (4, 64, True, 8, 8192, 8192, "tmem"), (4, 128, True, 8, 14336, 4096, "tmem"),
    (4, 128, True, 8, 25292, 2688, "i8mma"), (8, 128, True, 5, 28672, 2048, "i8mma"), (8, 128, True, 6, 28672, 2048, "tmem"),
    # the split-activation kernel from 100 MB, at two tokens from 115
    (4, -1, False, 2, 24576, 8192, "i8mma"), (4, -1, False, 3, 24576, 8192, "i8tc"), (4, -1, False, 2, 28672, 8192, "i8tc"),
    (4, 384, False, 10, 33024, 4224, "tmem"), (4, 64, False, 8, 14336, 4224, "i8mma"),
])
def test_choice(wbits, bs, zp, M, N, K, kernel):
  assert chosen(wbits, bs, zp, M, N, K) == kernel
  call, exact = call_and_exact(wbits, bs, zp, M, N, K, torch.bfloat16)
  assert qo.max_abs_rel(call(), exact) < 1e-2  # one rounding to bf16


@pytest.mark.parametrize("wbits,M,N,K,kernel", [
    (4, 128, 1024, 4096, "i8tc"), (4, 128, 1024, 8192, "tmem"), (4, 1008, 256, 512, "i8tc"), (4, 1009, 256, 512, "tmem"),
    (4, 84, 7168, 2048, "i8tc"), (4, 85, 7168, 2048, "tmem"), (4, 85, 7168, 1984, "i8tc"), (4, 200, 4096, 768, "tmem"),
    (8, 445, 2970, 1792, "i8tc"), (8, 445, 2970, 4096, "tmem"), (8, 1009, 2970, 1792, "tmem"), (8, 1009, 4112, 512, "i8tc"),
    (4, 8, 21601, 2208, "tmem"), (4, 5, 21601, 2208, "i8mma"), (8, 8, 21601, 2208, "tmem"), (8, 2, 14336, 4096, "i8mma"), (4, 8, 16384, 8192, "i8tc"),
])
def test_zero_points_per_channel(wbits, M, N, K, kernel):
  """Each line from both sides: few tokens, few items, long rows, more tokens than a launch of the split-activation kernel."""
  assert chosen(wbits, -1, True, M, N, K) == kernel
  for out_dtype, tol in ((torch.bfloat16, 1e-2), (torch.float32, 1e-5)):
    call, exact = call_and_exact(wbits, -1, True, M, N, K, out_dtype)
    # fp32: exact products or 2^-22 of the row's largest activation; sums of at most 512 products, then of those
    assert qo.max_abs_rel(call(), exact) < tol

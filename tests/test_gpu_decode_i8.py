"""The integer decode kernel against the CPU oracle at the sizes where its work split can go wrong: fewer tiles than CTAs,
ragged rows and columns, one to sixteen tokens (each number of MMA column tiles), scale blocks inside and across its
64-byte steps, more tiles than one CTA takes."""
import pytest
import torch

import xla_b200
from oracle import qmm_oracle as qo
from tests import qmm_cases as qc

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("with_zp", [False, True])
@pytest.mark.parametrize("wbits,bs,N,K,M", [
    (8, -1, 16, 64, 1), (8, -1, 261, 1056, 2), (8, 128, 40, 1280, 5), (8, 64, 777, 320, 8), (8, 256, 4096, 512, 3),
    (4, -1, 261, 1056, 1), (4, 128, 77, 4096, 4), (4, 64, 130, 192, 6), (4, 64, 33, 1984, 11), (4, 256, 16 * 148 * 8 + 3, 256, 2),
    (4, 128, 4099, 512, 16), (8, -1, 16 * 148 * 16 + 40, 128, 1), (8, -1, 300, 28672, 1),
])
def test_against_the_oracle(dtype, with_zp, wbits, bs, N, K, M):
  g = qc.gen(N + K + M)
  x = qc.activations(g, M, K, dtype, outliers=True)
  w = qc.int4_weight(g, N, K) if wbits == 4 else qc.int8_weight(g, N, K)
  s = qc.per_channel_scale(g, N) if bs == -1 else qc.blockwise_scale(g, K // bs, N)
  zp = torch.randint(-3, 4, s.shape, generator=g).float() * s if with_zp else None
  exact = qo.quantized_matmul(x.float(), w if bs == -1 else qc.to_sbn(w, bs), s, zp, block_size=bs, dot_round=None)
  wd = xla_b200.pack_int4(w.to(DEV)) if wbits == 4 else w.to(DEV)
  with xla_b200.force_variant("i8mma"):
    out = torch.ops.xla_b200.quantized_matmul_packed(x.to(DEV), wd, s.to(DEV), None if zp is None else zp.to(DEV), block_size=bs,
                                                     int4_weight=wbits == 4, weight_is_packed=wbits == 4, out_dtype=torch.float32)
  assert qo.max_abs_rel(out, exact) < 1e-5


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("with_zp", [False, True])
@pytest.mark.parametrize("M,N,K,kernel", [(1, 16, 64, b"i8mma"), (3, 261, 1072, b"i8mma"), (8, 4099, 512, b"i8mma"), (9, 130, 2048, b"i8mma"),
                                          (12, 77, 1040, b"i8mma"), (13, 300, 1040, b"tcgen05"), (17, 77, 144, b"tcgen05"),
                                          (32, 300, 256, b"tcgen05")])
def test_w8a8_equals_the_two_kernel_path(dtype, with_zp, M, N, K, kernel):
  """Quantization inside the decode kernel, up to twelve tokens, and the quantizer with the tensor-core GEMM from there on:
  the same bits as the quantizer kernel followed by the any-shape GEMM."""
  L = xla_b200._capi.lib()
  assert L.qmm_variant_for(xla_b200._capi.OP_W8A8_PERCHANNEL, M, N, K, 0, int(with_zp)) == kernel
  g = qc.gen(M + N + K)
  x = qc.activations(g, M, K, dtype, outliers=True).to(DEV)
  w, s = qc.int8_weight(g, N, K).to(DEV), qc.per_channel_scale(g, N).to(DEV)
  zp = (torch.randint(-20, 21, (N,), generator=g).float().to(DEV) * s) if with_zp else None
  for saturate in (True, False):
    xla_b200.set_activation_saturation(saturate)
    try:
      out = torch.ops.xla.quantized_matmul(x, w, s, zp, quantize_activation=True)
      with xla_b200.force_variant("generic"):
        ref = torch.ops.xla.quantized_matmul(x, w, s, zp, quantize_activation=True)
    finally:
      xla_b200.set_activation_saturation(True)
    assert torch.equal(out, ref)

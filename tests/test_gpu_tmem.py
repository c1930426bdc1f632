"""The tensor-memory kernel against the CPU oracle where its tiling can go wrong: every accumulator width, partial row and
token tiles, K that ends inside a step or a raw tile, items split over CTAs, scale blocks of 64 to several steps."""
import pytest
import torch

import xla_b200
from oracle import qmm_oracle as qo
from tests import qmm_cases as qc

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("wbits,bs,N,K,M", [
    (8, -1, 128, 64, 1), (8, -1, 300, 1056, 20), (8, 64, 130, 320, 33), (8, 128, 1000, 1280, 64), (8, 256, 129, 768, 65),
    (8, -1, 260, 2064, 128), (4, -1, 77, 4000, 16), (4, 128, 300, 1152, 50), (4, 64, 300, 1984, 40), (4, 64, 512, 192, 129),
    (4, 128, 128 * 149, 256, 130), (4, 256, 300, 1024, 193), (4, 128, 640, 4096, 400), (8, 512, 200, 1024, 577),
])
def test_against_the_oracle(dtype, wbits, bs, N, K, M):
  g = qc.gen(N + K + M)
  x = qc.activations(g, M, K, dtype, outliers=True)
  w = qc.int4_weight(g, N, K) if wbits == 4 else qc.int8_weight(g, N, K)
  s = qc.per_channel_scale(g, N) if bs == -1 else qc.blockwise_scale(g, K // bs, N)
  rows = torch.tensor(sorted({0, M // 3, M // 2, M - 2 if M > 1 else 0, M - 1}))
  exact = qo.quantized_matmul(x[rows].float(), w if bs == -1 else qc.to_sbn(w, bs), s, block_size=bs, dot_round=None)
  wd = xla_b200.pack_int4(w.to(DEV)) if wbits == 4 else w.to(DEV)
  with xla_b200.force_variant("tmem"):
    out = torch.ops.xla_b200.quantized_matmul_packed(x.to(DEV), wd, s.to(DEV), block_size=bs, int4_weight=wbits == 4,
                                                     weight_is_packed=wbits == 4, out_dtype=torch.float32)
  assert qo.max_abs_rel(out[rows.to(DEV)], exact) < 1e-5


@pytest.mark.parametrize("M", [65, 200, 1100])
def test_gate_up(M):
  g = qc.gen(M)
  N, K, bs = 128 * 101, 512, 128
  x = qc.activations(g, M, K)
  wg, wu = qc.int4_weight(g, N // 2, K), qc.int4_weight(g, N // 2, K)
  sg, su = qc.blockwise_scale(g, K // bs, N // 2), qc.blockwise_scale(g, K // bs, N // 2)
  w, s = xla_b200.interleave_gate_up(xla_b200.pack_int4(wg.to(DEV)), xla_b200.pack_int4(wu.to(DEV)), sg.to(DEV), su.to(DEV), bs)
  rows = torch.tensor([0, M // 2, M - 1])
  gate = qo.quantized_matmul(x[rows].float(), qc.to_sbn(wg, bs), sg, block_size=bs, dot_round=None)
  up = qo.quantized_matmul(x[rows].float(), qc.to_sbn(wu, bs), su, block_size=bs, dot_round=None)
  out = torch.ops.xla_b200.quantized_gate_up(x.to(DEV), w, s, block_size=bs, int4_weight=True, weight_is_packed=True,
                                             out_dtype=torch.float32)
  assert qo.max_abs_rel(out[rows.to(DEV)], torch.nn.functional.silu(torch.as_tensor(gate)) * torch.as_tensor(up)) < 1e-4


@pytest.mark.parametrize("wbits,M", [(4, 16), (8, 29), (4, 65), (8, 200)])
def test_gate_up_with_blocks_of_64(wbits, M):
  """The C ABI's fused form with scale blocks of 64 (the operator runs two steps there): up to 32 tokens on the split-activation
  kernel, above on the tensor-memory kernel."""
  from xla_b200 import _capi
  L = _capi.lib()
  g = qc.gen(M)
  N, K, bs = 640, 1024, 64
  weight = qc.int4_weight if wbits == 4 else qc.int8_weight
  x, wg, wu = qc.activations(g, M, K), weight(g, N, K), weight(g, N, K)
  sg, su = qc.blockwise_scale(g, K // bs, N) / 16, qc.blockwise_scale(g, K // bs, N)
  to_device = lambda w: xla_b200.pack_int4(w.to(DEV)) if wbits == 4 else w.to(DEV)  # noqa: E731
  w, s = xla_b200.interleave_gate_up(to_device(wg), to_device(wu), sg.to(DEV), su.to(DEV), bs)
  xd, out = x.to(DEV), torch.empty(M, N, device=DEV)
  nbytes = L.qmm_weight_only_workspace_size(M, K)
  ws = torch.zeros(nbytes, dtype=torch.uint8, device=DEV)
  with torch.cuda.device(0):
    _capi.check(L.qmm_gate_up(wbits, xd.data_ptr(), _capi.BF16, w.data_ptr(), s.data_ptr(), out.data_ptr(), _capi.F32, M, 2 * N, K, bs,
                              ws.data_ptr(), nbytes, _capi.stream_ptr(DEV)))
  gate = torch.as_tensor(qo.quantized_matmul(x.float(), qc.to_sbn(wg, bs), sg, block_size=bs, dot_round=None))
  up = torch.as_tensor(qo.quantized_matmul(x.float(), qc.to_sbn(wu, bs), su, block_size=bs, dot_round=None))
  assert qo.max_abs_rel(out, torch.nn.functional.silu(gate) * up) < 1e-4


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("wbits,bs,N,K,M", [
    (4, -1, 256, 512, 20), (8, -1, 256, 640, 20), (4, 128, 256, 384, 33), (8, 128, 256, 640, 64), (4, 64, 256, 192, 7),
    (8, 64, 256, 448, 64), (4, 128, 256, 896, 70), (8, 128, 256, 640, 150),
])
def test_every_weight_value_is_converted_exactly(dtype, wbits, bs, N, K, M):
  """Small whole activations and scales of one: the fp32 result is a whole number, equal to the integer product."""
  g = qc.gen(K + M)
  lo, hi = (-8, 8) if wbits == 4 else (-128, 128)
  w = (torch.arange(N * K, dtype=torch.int32).reshape(N, K) * 7 % (hi - lo) + lo).to(torch.int8)
  x = torch.randint(-2, 3, (M, K), generator=g)
  s = torch.ones((N,) if bs == -1 else (K // bs, N))
  wd = xla_b200.pack_int4(w.to(DEV)) if wbits == 4 else w.to(DEV)
  with xla_b200.force_variant("tmem"):
    out = torch.ops.xla_b200.quantized_matmul_packed(x.to(dtype).to(DEV), wd, s.to(DEV), block_size=bs, int4_weight=wbits == 4,
                                                     weight_is_packed=wbits == 4, out_dtype=torch.float32)
  assert torch.equal(out.cpu().long(), x.long() @ w.long().T)


@pytest.mark.parametrize("scales", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("zp", [False, True])
@pytest.mark.parametrize("wbits,bs,N,K,M", [
    (4, 128, 128 * 150 + 2, 640, 2), (4, 128, 1026, 1152, 32), (4, 128, 1026, 2176, 64), (8, 128, 514, 896, 31),
    (8, 128, 1026, 1408, 63), (4, 64, 514, 320, 32), (8, 64, 514, 832, 61), (4, 256, 514, 2304, 48), (8, 384, 514, 1152, 30),
    (4, 128, 514, 1920, 100), (4, 128, 514, 1920, 190), (8, -1, 514, 1136, 40), (4, -1, 514, 2592, 25),
])
def test_steps_that_the_blocks_do_not_fill(wbits, bs, N, K, M, zp, scales):
  """Odd numbers of scale blocks in steps of two, more tiles than CTAs, ragged rows; zero points; scales in the activations' type."""
  g = qc.gen(N + K + M)
  x = qc.activations(g, M, K, torch.bfloat16, outliers=True)
  w = qc.int4_weight(g, N, K) if wbits == 4 else qc.int8_weight(g, N, K)
  s = (qc.per_channel_scale(g, N) if bs == -1 else qc.blockwise_scale(g, K // bs, N)).to(scales)
  z = (torch.randint(-2, 3, s.shape, generator=g) * s).to(scales) if zp else None
  wd = xla_b200.pack_int4(w.to(DEV)) if wbits == 4 else w.to(DEV)
  with xla_b200.force_variant("tmem"):
    out = torch.ops.xla_b200.quantized_matmul_packed(x.to(DEV), wd, s.to(DEV), None if z is None else z.to(DEV), block_size=bs,
                                                     int4_weight=wbits == 4, weight_is_packed=wbits == 4, out_dtype=torch.float32)
  S = 1 if bs == -1 else K // bs
  xb, wb = x.double().to(DEV).view(M, S, K // S), w.double().to(DEV).view(N, S, K // S)
  exact = torch.einsum("msk,nsk,sn->mn", xb, wb, s.double().to(DEV).view(S, N))
  if zp:
    exact -= torch.einsum("ms,sn->mn", xb.sum(-1), z.double().to(DEV).view(S, N))
  # exact products, at most K / 128 + 3 roundings of the running sum: far below 1e-5 of the largest result
  assert qo.max_abs_rel(out, exact) < 1e-5


@pytest.mark.parametrize("wbits,bs,M", [(4, 128, 9), (4, 128, 32), (8, 128, 4), (4, 64, 20), (8, -1, 17)])
def test_gate_up_of_small_batches_on_large_weights(wbits, bs, M):
  """Where the operator takes the tensor-core form at up to 32 tokens: against the two projections and the activation."""
  from xla_b200 import _capi
  g = torch.Generator(device=DEV).manual_seed(M)
  N2, K = 9216, 4096
  assert _capi.lib().qmm_gate_up_on_tensor_cores(wbits, _capi.BF16, _capi.BF16, M, N2, K, max(bs, 0))
  w = torch.randint(0, 256, (N2, K * wbits // 8), generator=g, device=DEV, dtype=torch.uint8)
  w = w if wbits == 4 else w.view(torch.int8)
  s = (torch.rand((N2,) if bs == -1 else (K // bs, N2), generator=g, device=DEV) + 0.5) / (4.6 if wbits == 4 else 73.) / K**0.5
  x = torch.randn(M, K, generator=g, device=DEV).bfloat16()
  kw = dict(block_size=bs, int4_weight=wbits == 4, weight_is_packed=wbits == 4)
  out = torch.ops.xla_b200.quantized_gate_up(x, w, s, out_dtype=torch.bfloat16, **kw)
  y = torch.ops.xla_b200.quantized_matmul_packed(x, w, s, None, out_dtype=torch.float32, **kw).view(M, N2 // 16, 2, 8).double()
  ref = (torch.nn.functional.silu(y[:, :, 0]) * y[:, :, 1]).reshape(M, N2 // 2)
  assert qo.max_abs_rel(out, ref) < 1e-2  # one rounding to bf16


@pytest.mark.parametrize("wbits,bs,N,K,M", [
    (4, 384, 1030, 3840, 20), (8, 384, 1030, 3840, 64), (4, 384, 20000, 1536, 33), (8, 384, 514, 4224, 100), (4, 384, 514, 4224, 128),
    (8, -1, 514, 384, 100), (8, -1, 514, 704, 128), (8, -1, 514, 1152, 65), (8, 640, 514, 3840, 50), (4, 256, 514, 4096, 100),
])
def test_folds_of_several_steps(wbits, bs, N, K, M):
  """Three and five steps per fold, which one issuer has to itself, and two, which alternate: the same bits each time."""
  g = qc.gen(N + K + M)
  x = qc.activations(g, M, K, torch.bfloat16, outliers=True).to(DEV)
  w = (qc.int4_weight if wbits == 4 else qc.int8_weight)(g, N, K).to(DEV)
  s = (qc.per_channel_scale(g, N) if bs == -1 else qc.blockwise_scale(g, K // bs, N)).to(DEV)
  wd = xla_b200.pack_int4(w) if wbits == 4 else w
  with xla_b200.force_variant("tmem"):
    run = lambda: torch.ops.xla_b200.quantized_matmul_packed(x, wd, s, block_size=bs, int4_weight=wbits == 4,  # noqa: E731
                                                             weight_is_packed=wbits == 4, out_dtype=torch.float32)
    out = run()
    assert all(torch.equal(run(), out) for _ in range(5))
  S = 1 if bs == -1 else K // bs
  exact = torch.einsum("msk,nsk,sn->mn", x.double().view(M, S, -1), w.double().view(N, S, -1), s.double().view(S, N))
  assert qo.max_abs_rel(out, exact) < 1e-5  # exact products, a rounding per block and per 512 values


GATE_UP_ROUTES = [
    # from 100 MB at two to sixteen tokens: the split-activation kernel's narrow instances, of 16, 32 and 48 columns
    (4, 128, 2, 57344, 4096, "i8tc"), (4, 128, 5, 57344, 4096, "i8tc"), (4, 128, 6, 57344, 4096, "i8tc"), (4, 128, 10, 57344, 4096, "i8tc"),
    (8, -1, 16, 28672, 4096, "i8tc"), (4, -1, 13, 57344, 4096, "i8tc"),
    (4, 128, 10, 28672, 3072, "i8tc"), (4, 128, 11, 28672, 3072, "tmem"),
    # scale blocks that are a multiple of 128, but not of 256
    (4, 384, 9, 14336, 4224, "tmem"), (8, 384, 4, 14336, 4224, "tmem"),
]
LARGE_GATE_UP = """
import sys, torch, xla_b200
from xla_b200 import _capi
wbits, bs, M, N2, K = map(int, sys.argv[1:])
g = torch.Generator(device="cuda:0").manual_seed(M)
w = torch.randint(0, 256, (N2, K * wbits // 8), generator=g, device="cuda:0", dtype=torch.uint8)
w = w if wbits == 4 else w.view(torch.int8)
s = (torch.rand((N2,) if bs == -1 else (K // bs, N2), generator=g, device="cuda:0") + 0.5) / (4.6 if wbits == 4 else 73.) / K**0.5
x = torch.randn(M, K, generator=g, device="cuda:0").bfloat16()
kw = dict(block_size=bs, int4_weight=wbits == 4, weight_is_packed=wbits == 4)
out = torch.ops.xla_b200.quantized_gate_up(x, w, s, out_dtype=torch.float32, **kw)
with xla_b200.force_variant("generic"):
  y = torch.ops.xla_b200.quantized_matmul_packed(x, w, s, None, out_dtype=torch.float32, **kw).view(M, N2 // 16, 2, 8).double()
ref = (torch.nn.functional.silu(y[:, :, 0]) * y[:, :, 1]).reshape(M, N2 // 2)
print("error", float((out - ref).abs().max() / ref.abs().max()))
"""


@pytest.mark.parametrize("wbits,bs,M,N2,K,kernel", GATE_UP_ROUTES)
def test_gate_up_takes_the_kernel_it_asked_for(wbits, bs, M, N2, K, kernel):
  """The kernel by the library's log, in a process of its own, and the result against the any-shape kernel's two projections."""
  import os
  import subprocess
  import sys
  r = subprocess.run([sys.executable, "-c", LARGE_GATE_UP] + [str(v) for v in (wbits, bs, M, N2, K)], text=True, capture_output=True,
                     env=dict(os.environ, QMM_B200_LOG="1"), timeout=300, cwd=os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
  assert r.returncode == 0, r.stderr[-2000:]
  assert f"gate_up M={M} N={N2} K={K} -> {kernel}\n" in r.stderr, r.stderr[-500:]
  # exact products or three limbs: a rounding per block and K ones of the fp32 sums on either side, 2^-24 each at random
  assert float(r.stdout.split()[-1]) < 1e-5

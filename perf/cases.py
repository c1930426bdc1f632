"""The work that users of the quantized linear have it do, as cases that can be timed.

A case is a dict of plain values.  `work_kind` says what one pass is:

  linear   one quantized linear through one of the public entry points (`entry`):
             "op"      torch.ops.xla.quantized_matmul, weights as the reference holds them, fp32 scales
             "int8"    torch.ops.xla.quantized_matmul_int8, output in the activations' type
             "packed"  torch.ops.xla_b200.quantized_matmul_packed, K-minor weights, int4 two per byte
             "module"  XlaQuantizedLinear, scales in the activations' type (what quantizing a model of that type gives)
  layer    the seven linears of a decoder layer (q, k, v, o, gate, up, down) as XlaQuantizedLinear modules, int8 per channel
  mlp      a gated MLP with int4 block-128 weights: the fused gate/up operator, then the down projection

`m` tokens; `n` outputs, `k` inputs (linear) or `hidden` and `inter` sizes (layer, mlp).  `block` is the scale block along
K, -1 per channel; `zp`: asymmetric weights; `qact`: per-token dynamic int8 activations (W8A8).

Activations are N(0,1) with one entry in a hundred twenty times larger, as hidden states have them; weights are uniform
integers over their range; scales make the outputs of order one.
"""
import math

import torch

import xla_b200

_DTYPES = {"bf16": torch.bfloat16, "f16": torch.float16, "f32": torch.float32}
_FLOPS_MOST = 8e11  # no drawn case costs more than the largest listed one
_BYTES_MOST = 4e8


def _linear(entry, m, n, k, wbits=8, block=-1, zp=False, qact=False, x="bf16"):
  return {"work_kind": "linear", "entry": entry, "m": m, "n": n, "k": k, "wbits": wbits, "block": block, "zp": zp, "qact": qact,
          "x": x}


def listed():
  return [
      # one token through a square projection: the smallest call a decode loop makes, all latency
      dict(_linear("op", 1, 4096, 4096), name="op_w8_m1"),
      # the per-channel int8 configuration of the benchmark: sixteen sequences decoding together, fp32 result
      dict(_linear("op", 16, 4096, 4096), name="op_w8_m16"),
      # the int4 decode configuration of the benchmark, packed weights, eight sequences
      dict(_linear("packed", 8, 14336, 4096, wbits=4, block=128), name="packed_w4_block128_m8"),
      # asymmetric int4 (the module's default is asymmetric) in fp16, an odd number of sequences, a wide fused projection
      dict(_linear("module", 29, 37888, 3584, wbits=4, block=128, zp=True, x="f16"), name="module_w4_block128_zp_m29_f16"),
      # fp32 activations, asymmetric int8, a prompt of a ragged length
      dict(_linear("op", 333, 5120, 6912, zp=True, x="f32"), name="op_w8_zp_m333_f32"),
      # W8A8 in a decode loop: four sequences, a module with dynamic activation quantization
      dict(_linear("module", 4, 14336, 4096, qact=True), name="module_w8a8_m4"),
      # W8A8 prefill: the benchmark's configuration
      dict(_linear("int8", 2048, 4096, 4096, qact=True), name="int8_w8a8_m2048"),
      # a whole 8B-shaped decoder layer, one sequence decoding: seven calls that depend on the weight stream
      {"work_kind": "layer", "m": 1, "hidden": 4096, "inter": 14336, "x": "bf16", "name": "layer8b_m1"},
      # the same layer on a prompt
      {"work_kind": "layer", "m": 512, "hidden": 4096, "inter": 14336, "x": "bf16", "name": "layer8b_m512"},
      # the 70B-shaped MLP of the benchmark: one sequence, a decode batch, a prompt
      {"work_kind": "mlp", "m": 1, "hidden": 8192, "inter": 28672, "x": "bf16", "name": "mlp70b_m1"},
      {"work_kind": "mlp", "m": 64, "hidden": 8192, "inter": 28672, "x": "bf16", "name": "mlp70b_m64"},
      {"work_kind": "mlp", "m": 512, "hidden": 8192, "inter": 28672, "x": "bf16", "name": "mlp70b_m512"},
  ]


def _log_int(rng, lo, hi):
  return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_once(rng):
  kind = rng.choice(("linear", "linear", "linear", "linear", "layer", "mlp"))
  x = rng.choice(("bf16", "bf16", "bf16", "f16", "f16", "f32"))
  if kind != "linear":
    # whole layers and MLPs of models from 1B to 70B, 16-bit activations
    hidden = 256 * _log_int(rng, 4, 32)
    inter = 256 * int(hidden * rng.uniform(2.0, 3.6) / 256)
    return {"work_kind": kind, "m": _log_int(rng, 1, 1024), "hidden": hidden, "inter": inter, "x": "bf16" if x == "f32" else x}
  # any output count (vocabularies and shards are odd), inputs in multiples of a scale block or a ragged multiple of 32
  m, n = _log_int(rng, 1, 8192), _log_int(rng, 256, 40000)
  entry = rng.choice(("op", "int8", "packed", "packed", "module", "module"))
  wbits, block, zp, qact = 8, -1, False, False
  if entry == "int8":
    qact = rng.random() < 0.5
  elif entry == "op":
    zp, qact = rng.random() < 0.3, rng.random() < 0.25
  else:
    wbits = rng.choice((4, 4, 8))
    block = rng.choice((-1, 64, 128, 128, 128, 256))
    zp = rng.random() < 0.3
  unit = 256 if block == -1 else block
  k = unit * max(1, round(_log_int(rng, 512, 28672) / unit))
  if block == -1 and rng.random() < 0.25:
    k += 32 * rng.randint(1, 7)
  return _linear(entry, m, n, k, wbits, block, zp, qact, x)


def draw(rng):
  while True:
    case = _draw_once(rng)
    w = work(case)
    if w["flops"] <= _FLOPS_MOST and w["bytes"] <= _BYTES_MOST:
      return case


# ---- inputs ------------------------------------------------------------------------------------------------------------


def _activations(g, m, k, dtype):
  x = torch.randn(m, k, generator=g, device="cuda")
  large = torch.rand(m, k, generator=g, device="cuda") < 0.01
  return torch.where(large, x * 20.0, x).to(dtype)


def _int_weight(g, shape, wbits):
  lo, hi = (-8, 8) if wbits == 4 else (-127, 128)
  return torch.randint(lo, hi, shape, generator=g, device="cuda", dtype=torch.int8)


def _scale(g, shape, k, wbits):
  spread = 4.6 if wbits == 4 else 73.0  # standard deviation of the uniform integers
  return (torch.rand(shape, generator=g, device="cuda") + 0.5) / (spread * math.sqrt(k))


def _zero_point(g, scale, wbits):
  most = 2 if wbits == 4 else 20
  return torch.randint(-most, most + 1, scale.shape, generator=g, device="cuda").float() * scale


def _module(g, n, k, wbits, block, zp, qact, dtype):
  mod = xla_b200.XlaQuantizedLinear(k, n, is_symmetric=not zp, block_size=block, int4_weight=wbits == 4,
                                    quantize_activation=qact)
  w = _int_weight(g, (n, k) if block == -1 else (k // block, block, n), wbits)
  s = _scale(g, (n,) if block == -1 else (k // block, n), k, wbits)
  mod.load_quantized_weight(w, s.to(dtype), _zero_point(g, s, wbits).to(dtype) if zp else None)
  return mod


def prepare(case, seed):
  g = torch.Generator(device="cuda").manual_seed(seed)
  dtype = _DTYPES[case["x"]]
  m = case["m"]
  if case["work_kind"] == "layer":
    h, i = case["hidden"], case["inter"]
    sizes = {"q": (h, h), "k": (h // 4, h), "v": (h // 4, h), "o": (h, h), "gate": (i, h), "up": (i, h), "down": (h, i)}
    mods = {name: _module(g, n, k, 8, -1, False, False, dtype) for name, (n, k) in sizes.items()}
    return {"kind": "layer", "mods": mods, "x": _activations(g, m, h, dtype), "attn": _activations(g, m, h, dtype),
            "act": _activations(g, m, i, dtype)}
  if case["work_kind"] == "mlp":
    h, i = case["hidden"], case["inter"]
    bytes4 = lambda n, k: torch.randint(0, 256, (n, k // 2), generator=g, device="cuda", dtype=torch.uint8)  # noqa: E731
    w_gu, s_gu = xla_b200.interleave_gate_up(bytes4(i, h), bytes4(i, h), _scale(g, (h // 128, i), h, 4),
                                             _scale(g, (h // 128, i), h, 4), block_size=128)
    return {"kind": "mlp", "x": _activations(g, m, h, dtype), "gate_up": w_gu, "gate_up_scale": s_gu, "down": bytes4(h, i),
            "down_scale": _scale(g, (i // 128, h), i, 4), "dtype": dtype}
  n, k, wbits, block, zp, qact = (case[f] for f in ("n", "k", "wbits", "block", "zp", "qact"))
  state = {"kind": case["entry"], "x": _activations(g, m, k, dtype), "block": block, "qact": qact, "dtype": dtype, "wbits": wbits}
  if case["entry"] == "module":
    state["mod"] = _module(g, n, k, wbits, block, zp, qact, dtype)
    return state
  if case["entry"] == "packed" and wbits == 4:
    state["w"] = torch.randint(0, 256, (n, k // 2), generator=g, device="cuda", dtype=torch.uint8)
  else:
    state["w"] = _int_weight(g, (n, k), wbits)
  state["s"] = _scale(g, (n,) if block == -1 else (k // block, n), k, wbits)
  state["zp"] = _zero_point(g, state["s"], wbits) if zp else None
  return state


def run(state):
  kind, x = state["kind"], state["x"]
  if kind == "op":
    return torch.ops.xla.quantized_matmul(x, state["w"], state["s"], state["zp"], quantize_activation=state["qact"])
  if kind == "int8":
    return torch.ops.xla.quantized_matmul_int8(x, state["w"], state["s"], quantize_activation=state["qact"])
  if kind == "packed":
    return torch.ops.xla_b200.quantized_matmul_packed(x, state["w"], state["s"], state["zp"], block_size=state["block"],
                                                      int4_weight=state["wbits"] == 4, weight_is_packed=state["wbits"] == 4,
                                                      out_dtype=state["dtype"])
  if kind == "module":
    return state["mod"](x)
  if kind == "layer":
    mods = state["mods"]
    return [mods["q"](x), mods["k"](x), mods["v"](x), mods["o"](state["attn"]), mods["gate"](x), mods["up"](x),
            mods["down"](state["act"])]
  h = torch.ops.xla_b200.quantized_gate_up(x, state["gate_up"], state["gate_up_scale"], block_size=128, int4_weight=True,
                                           weight_is_packed=True, out_dtype=state["dtype"])
  return torch.ops.xla_b200.quantized_matmul_packed(h, state["down"], state["down_scale"], block_size=128, int4_weight=True,
                                                    weight_is_packed=True, out_dtype=state["dtype"])


# ---- what a pass cannot do without ------------------------------------------------------------------------------------


def _out_bytes(case):
  # operators given fp32 scales return fp32 by type promotion; the others return the activations' type
  return 4 if case["x"] == "f32" or case.get("entry") == "op" else 2


def _linear_work(m, n, k, wbits, block, zp, xbytes, obytes, sbytes):
  scales = n * (1 if block == -1 else k // block) * (2 if zp else 1)
  return m * k * xbytes + n * k * wbits / 8 + scales * sbytes + m * n * obytes, 2.0 * m * n * k


def work(case):
  m, xb = case["m"], 4 if case["x"] == "f32" else 2
  if case["work_kind"] == "layer":
    h, i = case["hidden"], case["inter"]
    w = h * h * 2 + 2 * (h // 4) * h + 3 * h * i
    outs = 2 * h + 2 * (h // 4) + 2 * i + h
    return {"bytes": w + xb * outs + m * (2 * h + i) * xb + m * outs * xb, "flops": 2.0 * m * w}
  if case["work_kind"] == "mlp":
    h, i = case["hidden"], case["inter"]
    w = 3 * h * i
    return {"bytes": w / 2 + 4 * (w // 128) + 2 * m * h * xb, "flops": 2.0 * m * w}
  sb = xb if case["entry"] == "module" else 4
  b, f = _linear_work(m, case["n"], case["k"], case["wbits"], case["block"], case["zp"], xb, _out_bytes(case), sb)
  return {"bytes": b, "flops": f}


def tolerance(case):
  if case["work_kind"] == "linear" and case["qact"]:
    return "exact"  # integer products and sums, and one defined order of the fp32 products after them
  if _out_bytes(case) == 4 and case["work_kind"] == "linear":
    return {"rel": 3e-5}
  return {"rel": 6e-3 if case["x"] == "bf16" else 1e-3}

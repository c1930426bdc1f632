"""The rule that lets the tensor-memory GEMM's two MMA issuers alternate, against a model of the barriers on the CPU."""
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "xla_b200", "csrc")
FOLDS = range(1, 13)
# (operand slots, activation stages) of the kernel's instances, and a few others
RINGS = [(4, 4), (2, 4), (4, 8), (2, 8), (2, 3), (4, 6), (2, 2), (4, 3), (3, 5)]


def acc_last(a_slots, b_slots):
  return a_slots % 2 == 0 and b_slots % 2 == 0


def first_early_wait(fu, a_slots, b_slots, alternate, steps=96):
  """The first step whose wait could be taken for the phase before, or None.  Events know what happened before them: a wait knows its
  barrier's phase, the MMAs of a step its waits, a drained fold its MMAs and the fold before, an operand slot the MMAs that read it last.
  A parity wait for step j needs to know, before it looks, of the phase of step j - ring."""
  issuer_knows = [set(), set()]
  mma, drained = {}, {}
  for j in range(steps):  # an order in which everything that an event knows of comes before it
    fold, q = divmod(j, fu)
    me = issuer_knows[fold % 2 if alternate else 0]
    accumulator = lambda: me.update(drained[fold - 2]) if q == 0 and fold >= 2 else None  # noqa: E731
    if not acc_last(a_slots, b_slots):
      accumulator()
    for ring, n in (("b", b_slots), ("a", a_slots)):
      if j >= n and (ring, j - n) not in me:
        return j
      me.add((ring, j))
      me.update(mma.get(j - n, ()))  # the producer filled the slot after the MMAs of step j - n
    if acc_last(a_slots, b_slots):
      accumulator()
    mma[j] = frozenset(me)
    if q == fu - 1:
      drained[fold] = mma[j] | drained.get(fold - 1, frozenset())
  return None


@pytest.fixture(scope="module")
def rule(tmp_path_factory):
  exe = str(tmp_path_factory.mktemp("rule") / "rule")
  src = """#include <cstdio>
#include "issue_order.h"
int main() { int f, a, b, l; while (scanf("%d %d %d %d", &f, &a, &b, &l) == 4) printf("%d\\n", (int)qmm::issuers_may_alternate(f, a, b, l)); }
"""
  subprocess.run([os.environ.get("CXX", "g++"), "-std=c++17", f"-I{CSRC}", "-x", "c++", "-", "-o", exe], input=src, text=True, check=True)
  asked = [(fu, a, b) for fu in FOLDS for a, b in RINGS]
  lines = "".join(f"{fu} {a} {b} {int(acc_last(a, b))}\n" for fu, a, b in asked)
  got = subprocess.run([exe], input=lines, text=True, check=True, capture_output=True).stdout.split()
  return {k: v == "1" for k, v in zip(asked, got, strict=True)}


@pytest.mark.parametrize("a_slots,b_slots", RINGS)
@pytest.mark.parametrize("fu", FOLDS)
def test_no_wait_comes_a_phase_early(rule, fu, a_slots, b_slots):
  assert first_early_wait(fu, a_slots, b_slots, alternate=False) is None
  if rule[fu, a_slots, b_slots]:
    assert first_early_wait(fu, a_slots, b_slots, alternate=True) is None


def test_the_model_sees_early_waits_and_the_rule_keeps_the_common_folds(rule):
  # three steps per fold (scale blocks of 384): steps of the other issuer lie between a slot's turns
  assert first_early_wait(3, 4, 4, True) is not None and first_early_wait(3, 4, 8, True) is not None
  assert all(rule[1, a, b] for a, b in RINGS if a % 2 == 0) and rule[2, 4, 4] and rule[2, 4, 8]

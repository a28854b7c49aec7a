"""The bits of the step: in every kernel class, the fields after two steps from
a random state are those of the golden file.  The error bounds of the other
tests do not see a sum in another order or a product contracted into another
one; 16-bit storage does, for they decide which stored values round up, and a
run continued with such a build departs from itself by up to 6e-4 in twenty
steps (bfloat16)."""
import json
import os

import pytest

import step_bits

pytestmark = pytest.mark.gpu

with open(os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden", "step_bits.json")) as _f:
    GOLDEN = json.load(_f)


@pytest.mark.parametrize("storage", ["f32", "f16", "bf16", "f64"])
def test_fields_after_two_steps(storage):
    mine = {step_bits.name(c): step_bits.crc(c) for c in step_bits.classes() if c[0] == storage}
    assert mine and [n for n, v in mine.items() if v != GOLDEN[n]] == []

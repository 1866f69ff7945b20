"""No plan runs longer FP32 chains than the recorded ones (host only).

The golden spans are those the K-split rule of csrc/chains.cpp gives, recorded
when the rule was the planner itself.  Time models may move a plan to another
engine, tile or a finer split; never to a longer chain, and never from plain
FP32 to a tensor-core form."""
import json
import os

import pytest

with open(os.path.join(os.path.dirname(__file__), "golden", "chain_spans.json")) as f:
    SPANS = json.load(f)


@pytest.mark.parametrize("col,engine", [(3, "auto"), (4, "packed"), (5, "onchip")])
def test_products(cg3m, col, engine):
    longer = [(row, p) for row in SPANS["product"]
              if (p := cg3m.plan("N", "N", *row[:3], alpha=0.5, engine=engine))["k_span"] > row[col]]
    assert not longer


def test_onchip_family(cg3m):
    longer = [(row, p) for row in SPANS["onchip"] if (p := cg3m.plan_onchip(*row[:5]))["k_span"] > row[5]]
    assert not longer


def test_tensor_forms(cg3m):
    """Recorded as plain FP32: still plain FP32, no longer chains.  Recorded as
    the form: that form (its error does not depend on the split), or FP32 chains
    within the segments it accumulates."""
    for m, n, k, form, tensor, span in SPANS["tensor"]:
        p = cg3m.plan("N", "N", m, n, k, alpha=0.5, form=form)
        segment = 128 if k >= 2048 else 64 if k > 1024 else 32
        if not tensor:
            assert p["form"] == cg3m.FORM["fp32"] and p["k_span"] <= span, (m, n, k, form)
        elif p["form"] == cg3m.FORM["fp32"]:
            assert p["k_span"] <= segment, (m, n, k, form)


# 204 and 213 terms: four partitions of 64 took 19.9 us, two of 128 23.8 (3xTF32)
@pytest.mark.parametrize("m,n,k", [(546, 739, 204), (535, 704, 213)])
def test_short_tensor_products_split_four_ways(cg3m, m, n, k):
    assert cg3m.plan("N", "N", m, n, k, alpha=0.5, form="tf32x3", engine="packed")["k_partitions"] == 4

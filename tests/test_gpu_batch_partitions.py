"""Batches that are not timed keep the K partitions of the split rule
(csrc/chains.cpp), whatever tiles they take."""
import json
import os

import pytest

pytestmark = pytest.mark.gpu

# [m, n, k, partitions] of every problem of a batch, recorded when the rule's
# own tiles were used
with open(os.path.join(os.path.dirname(__file__), "golden", "batch_partitions.json")) as f:
    BATCHES = json.load(f)


@pytest.mark.parametrize("shapes", BATCHES, ids=[str(len(b)) for b in BATCHES])
def test_untuned_partitions(cg3m, cuda, shapes):
    import torch

    A, B = (torch.zeros(max(s[i] * s[2] for s in shapes), dtype=torch.complex64, device=cuda) for i in (0, 1))
    C = torch.zeros(sum(s[0] * s[1] for s in shapes), dtype=torch.complex64, device=cuda)
    problems, c = [], 0
    for m, n, k, _ in shapes:
        problems.append(("N", "N", m, n, k, 1.0, A, m, B, k, 0.0, C[c:], m))
        c += m * n
    plan = cg3m.default_handle().batch_plan(problems, tune=False)
    fewer = [(s, d) for s, d in zip(shapes, plan.describe()) if d[2] < s[3]]
    assert not fewer

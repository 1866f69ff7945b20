"""K splits keep FP32 chains short (host only).

A chain of t round-to-nearest FMAs leaves an error that grows as sqrt(t).  Up to
1024 terms a split is chosen for speed alone; beyond, the one-launch engine runs
chains at most twice as long as the packed engine's split (1.4 times its error),
narrow outputs with a clear gain excepted, and strided batches none longer than
a task of a quarter of an SM's work allows.
"""
import pytest

SHORT = 1024


@pytest.mark.parametrize("m,n,k", [
    (600, 1300, 1025), (600, 1300, 1646), (756, 344, 3425), (847, 32, 13564), (51, 460, 24997),
    (61, 734, 8372), (102, 253, 4429), (128, 128, 65536), (654, 1081, 784), (512, 512, 1024),
])
def test_product_chains(cg3m, m, n, k):
    auto = cg3m.plan("N", "N", m, n, k)
    packed = cg3m.plan("N", "N", m, n, k, engine="packed")
    assert auto["k_span"] <= max(SHORT, 2 * packed["k_span"])


@pytest.mark.parametrize("m,n,k", [(25, 1025, 59274), (25, 972, 13788), (1536, 24, 30000)])
def test_narrow_chains_take_fine_splits(cg3m, m, n, k):
    auto = cg3m.plan("N", "N", m, n, k)
    assert auto["k_partitions"] >= 7


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("m,n,k,batch,parts", [
    (22, 224, 1401, 8, 2), (401, 327, 3083, 5, 3), (452, 401, 7467, 4, 4), (32, 32, 1024, 4, 1), (512, 512, 4096, 64, 1),
])
def test_strided_chains(cg3m, m, n, k, batch, parts, mode):
    assert cg3m.plan_onchip(m, n, k, mode, batch)["k_partitions"] >= parts


@pytest.mark.parametrize("m,n,k", [(285, 52, 6745), (17, 159, 13980), (99, 29, 16878), (347, 29, 6625)])
def test_finer_splits_stay_in_a_default_workspace(cg3m, m, n, k):
    """Shapes whose planes and 32 partitions fit 32 MiB are not pushed past it."""
    assert cg3m.plan("N", "N", m, n, k)["workspace_bytes"] <= (32 << 20) - 256

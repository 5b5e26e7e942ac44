"""Which K splits the planner takes up to 16 tokens (CPU only, capacities of an imagined chip)."""
import pytest


@pytest.fixture(scope="module")
def capi(native_build):
    from hf_rocm_kernels import _capi

    return _capi


def _plan(capi, m, n, k, capacity):
    table = [[0, 0, 0, 0]] + [[0] + [148 * per_sm // split for per_sm in (1, 2, 3)] for split in range(1, 17)]
    for split, value in capacity.items():
        table[split] = [0, value // 3, value * 2 // 3, value]
    capi.override_device_model(148, table)
    try:
        return capi.plan(m, n, k)
    finally:
        capi.override_device_model(capacity=None)


@pytest.mark.parametrize("spare,split", [(1, 4), (2, 5)])
def test_two_clusters_stay_free(capi, spare, split):
    """81 tiles as clusters of 5 need room for 83; with less the next smaller split is taken."""
    none = {s: 0 for s in range(6, 17)}
    assert _plan(capi, 11, 10336, 6992, {**none, 5: 81 + spare, 4: 104})["split_k"] == split


@pytest.mark.parametrize("n,k,split", [(1104, 1104, 9), (1808, 1808, 9), (3360, 1984, 8)])
def test_one_k_block_per_cta_while_sms_are_idle(capi, n, k, split):
    """9 tiles x 9 K blocks and 15 x 9 CTAs fit on 148 SMs; 27 tiles do not, and keep two K blocks per CTA."""
    assert _plan(capi, 16, n, k, {})["split_k"] == split

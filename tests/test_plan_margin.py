"""Which K splits the planner takes up to 16 tokens (CPU only, capacities of an imagined chip)."""
import pytest


@pytest.fixture(scope="module")
def capi(native_build):
    from hf_rocm_kernels import _capi

    return _capi


def _plan(capi, m, n, k, capacity):
    """``capacity``: per split the clusters that fit with three CTAs on an SM, or (one, two, three) of them."""
    table = [[0, 0, 0, 0]] + [[0] + [148 * per_sm // split for per_sm in (1, 2, 3)] for split in range(1, 17)]
    for split, value in capacity.items():
        table[split] = [0, *value] if isinstance(value, tuple) else [0, value // 3, value * 2 // 3, value]
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


@pytest.mark.parametrize("m", [1, 4, 16])
@pytest.mark.parametrize("fit,shape", [(33, (8, 5)), (34, (8, 5)), (32, None)])
def test_a_measured_shape_needs_one_free_cluster(capi, m, fit, shape):
    """The 8B down projection was measured as 32 clusters of 8 at two CTAs per SM on chips that hold 33."""
    got = _plan(capi, m, 4096, 14336, {8: (16, fit, 50)})
    assert ((got["split_k"], got["num_stages"]) == (8, 5)) == (shape is not None)


@pytest.mark.parametrize("spare,split", [(0, 4), (1, 5), (2, 5)])
def test_one_cluster_stays_free_at_two_ctas_per_sm(capi, spare, split):
    """Two CTAs per SM (nothing larger than 5 fits, nothing at all at three per SM): 40 tiles need room for 41."""
    none = {s: (0, 0, 0) for s in (2, 3, *range(6, 17))}
    assert _plan(capi, 16, 5120, 9600, {**none, 4: (37, 74, 0), 5: (20, 40 + spare, 0)})["split_k"] == split


# (tiles, K blocks, split that needs all but one cluster, the next smaller one that fits with two to spare)
@pytest.mark.parametrize("tiles,k,split,smaller,two", [
    (30, 4096, 12, 10, True), (23, 12288, 15, 13, True),           # clusters of 11 and more
    (55, 2048, 7, 6, True), (47, 4096, 8, 7, True),                # 6 to 10, up to four K blocks per CTA
    (55, 4096, 7, 6, False), (47, 12288, 8, 7, False),             # more of them
    (103, 4096, 4, 3, False), (103, 12288, 4, 3, False)])          # up to 4
@pytest.mark.parametrize("m", [1, 16])
def test_how_many_clusters_stay_free(capi, m, tiles, k, split, smaller, two):
    for spare in (1, 2):
        capacity = {s: 0 for s in range(split + 1, 17)}
        capacity.update({s: tiles for s in range(smaller + 1, split)})     # full: never taken
        capacity.update({split: tiles + spare, smaller: 4 * tiles})
        got = _plan(capi, m, tiles * 128, k, capacity)["split_k"]
        assert got == (split if spare == 2 or not two else smaller)


@pytest.mark.parametrize("n,k,split", [
    (1104, 1104, 9), (848, 2032, 16),               # one K block per CTA
    (848, 2368, 16), (1808, 1808, 9),               # one or two, where half as many CTAs would have up to three
    (2416, 256, 1), (2360, 256, 2),                 # two in all, whole pieces of 16 rows and not
    (1400, 2256, 9), (1696, 1536, 6), (704, 4096, 16), (648, 3040, 12)])   # two each: no more CTAs for the same longest range
def test_more_ctas_only_for_a_shorter_range(capi, n, k, split):
    assert _plan(capi, 16, n, k, {})["split_k"] == split
    if split > 1 and -(-k // 128) % split == 0 and -(-k // 128) // split == 2:      # the split of two each does not fit: then more
        assert _plan(capi, 16, n, k, {split: 1})["split_k"] != split

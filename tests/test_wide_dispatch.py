"""Which kernel and which launch shape a call takes (CPU only, capacities of an imagined chip)."""
import pytest


@pytest.fixture(scope="module")
def capi(native_build):
    from hf_rocm_kernels import _capi

    return _capi


@pytest.fixture(autouse=True)
def chip(capi):
    """A chip whose GPCs hold 85 % of the clusters that the SM count allows."""
    table = [[0, 0, 0, 0]] + [[0] + [148 * p // s * (100 if s == 1 else 85) // 100 for p in (1, 2, 3)] for s in range(1, 17)]
    capi.override_device_model(148, table)
    yield
    capi.override_device_model(capacity=None)


CLUSTER, STREAMK, WIDE = 1, 2, 3


@pytest.mark.parametrize("n,k", [(4096, 4096), (28672, 4096), (17, 128), (8192, 28672)])
def test_more_than_64_tokens_run_wide_and_up_to_16_do_not(capi, n, k):
    for m in (1, 16):
        assert capi.launch_info(m, n, k)["kernel"] == CLUSTER
    for m in (65, 128, 129, 256, 257, 1000):
        info = capi.launch_info(m, n, k)
        assert info["kernel"] == WIDE
        launches = -(-m // 256)
        assert 0 <= info["m_pad"] - -(-m // launches) < 16     # the tokens of one launch, shared out evenly


def test_explicit_and_tuned_calls_stay_on_the_kernel_they_name(capi):
    for m in (65, 130, 256):
        assert capi.launch_info(m, 2000, 4096, split_k=3)["kernel"] == CLUSTER
        assert capi.launch_info(m, 2000, 4096, num_stages=4)["kernel"] == CLUSTER
        assert capi.launch_info(m, 2000, 4096, kernel=CLUSTER)["kernel"] == CLUSTER
        assert capi.launch_info(m, 2000, 4096, kernel=STREAMK)["kernel"] == STREAMK
    capi.lib.hfrk_tuning_set(64, 2000, 4096, 2, 3)
    try:
        info = capi.launch_info(130, 2000, 4096)
        assert (info["kernel"], info["split_k"], info["num_stages"]) == (CLUSTER, 2, 3)
        assert capi.launch_info(130, 2016, 4096)["kernel"] == WIDE
        assert capi.launch_info(130, 2000, 4096, kernel=WIDE)["kernel"] == WIDE
    finally:
        capi.lib.hfrk_tuning_clear()
    assert capi.launch_info(130, 2000, 4096)["kernel"] == WIDE


@pytest.mark.parametrize("m,kernel", [(1, CLUSTER), (16, CLUSTER), (17, WIDE), (64, WIDE), (65, WIDE), (300, WIDE)])
def test_swiglu_form(capi, m, kernel):
    assert capi.launch_info(m, 2048, 1024, form=2)["kernel"] == kernel


@pytest.mark.parametrize("swiglu", [False, True])
@pytest.mark.parametrize("m", [1, 17, 64, 128, 129, 200, 256])
def test_every_pinned_shape_keeps_its_bounds(capi, m, swiglu):
    """Ring, receive buffer and TMEM of every shape that the planner lets through, by the layouts of the kernel."""
    halves = 2 if m > 128 else 1
    rows = -(-(-(-m // halves)) // 8) * 8 * halves
    step = 32 if swiglu else 16
    for split in range(1, 9):
        for tile in range(32, 257, step):
            for stages in (2, 8):
                for per_sm in (1, 2):
                    out = (capi.ctypes.c_int * 8)()
                    rc = capi.lib.hfrk_gemm_launch_info(m, 2080, 2064, 2 * swiglu, WIDE, split, tile, stages, per_sm, out)
                    if rc != 0:
                        assert rc == 6
                        continue
                    kernel, got_split, got_stages, ctas, smem, m_pad, k_blocks, rows_w = list(out)
                    assert (kernel, got_split, m_pad, k_blocks, rows_w) == (WIDE, split, rows, 17, tile)
                    assert 2 <= got_stages <= stages and ctas == -(-2080 // tile) * split
                    ring = got_stages * (halves * 16384 + tile * 128)
                    groups = tile // step
                    assert groups >= split
                    if split > 1:
                        assert split * -(-groups // split) * step * (rows + 1) * 4 <= ring
                        assert ctas // split <= 148 * per_sm // split * 85 // 100
                    else:
                        assert 8 * 32 * 36 * 4 <= ring
                    columns = halves * max(32, 1 << (tile - 1).bit_length())
                    assert 1024 + ring < smem <= 227 * 1024 and per_sm * (smem + 1024) <= 228 * 1024
                    assert columns * per_sm <= 512 and (smem + 1024) * 512 >= columns * 228 * 1024 * 0.999


def test_bad_queries(capi):
    out = (capi.ctypes.c_int * 8)()
    for args in ((0, 128, 128, 0, 0), (16, 128, 128, 0, 4), (16, 127, 128, 2, 0), (16, 128, 128, 2, 1), (16, 128, 128, 3, 0), (300, 128, 128, 0, -1)):
        assert capi.lib.hfrk_gemm_launch_info(*args, 0, 0, 0, 0, out) == 6
    assert capi.lib.hfrk_gemm_launch_info(200, 128, 128, 0, WIDE, 9, 0, 0, 0, out) == 6       # more than eight CTAs per cluster
    assert capi.lib.hfrk_gemm_launch_info(200, 128, 128, 0, WIDE, 2, 0, 0, 0, out) == 6       # more than the K blocks
    assert capi.lib.hfrk_gemm_launch_info(200, 128, 128, 0, WIDE, 0, 40, 0, 0, out) == 6      # no multiple of 16
    assert capi.lib.hfrk_wide_gemm_fp8(0, 0, 0, 0, 0, 16, 128, 128, 128, 0, 0, 1, 0, 0, 0, 0, 0, 0, 0) == 6


ACCUMULATE, STORE = 0, 1


# The skinny kernel's plan on the chip above is part of the case: (split, rows per owner) by which the line is drawn.
@pytest.mark.parametrize("m,n,k,split,rows,accumulate,store", [
    (24, 4096, 4096, 7, 4, CLUSTER, CLUSTER),        # owners of up to eight rows
    (48, 6144, 4096, 7, 8, CLUSTER, CLUSTER),
    (24, 4096, 512, 2, 16, WIDE, CLUSTER),           # sixteen, up to 32 tokens: accumulating calls only
    (25, 17776, 4672, 2, 16, CLUSTER, CLUSTER),      # ... one long K range per wide CTA
    (21, 18527, 832, 2, 16, CLUSTER, CLUSTER),       # ... rows of D unaligned, tall tiles
    (21, 18528, 832, 2, 16, WIDE, CLUSTER),
    (64, 6144, 4096, 4, 16, WIDE, WIDE),             # 33 to 64 tokens: few tiles, full owners
    (44, 1288, 992, 4, 16, WIDE, CLUSTER),
    (33, 10544, 1568, 3, 16, WIDE, CLUSTER),
    (39, 11936, 8208, 3, 16, WIDE, WIDE),            # 94 tiles
    (49, 5760, 928, 4, 16, WIDE, WIDE),              # two K blocks per skinny CTA
    (41, 15435, 1344, 3, 16, CLUSTER, WIDE), (41, 15436, 1344, 3, 16, WIDE, WIDE),   # odd N on tall tiles
    (64, 14336, 4096, 2, 32, WIDE, WIDE), (54, 8192, 1024, 3, 32, WIDE, WIDE),   # 32 rows per owner
    (33, 28672, 4096, 1, 0, CLUSTER, CLUSTER),       # no split, one wave
    (30, 39840, 6272, 1, 0, WIDE, WIDE),             # a second wave that has hardly begun
    (30, 57344, 8192, 1, 0, CLUSTER, CLUSTER),       # one that is well filled, long K
    (30, 57344, 2048, 1, 0, WIDE, WIDE),
    (64, 57344, 8192, 1, 0, WIDE, WIDE),
])
def test_17_to_64_tokens(capi, m, n, k, split, rows, accumulate, store):
    plan = capi.launch_info(m, n, k, kernel=CLUSTER)
    assert plan["split_k"] == split
    if split > 1:
        assert 1 << (-(-m // split) - 1).bit_length() == rows
    assert capi.launch_info(m, n, k, ACCUMULATE)["kernel"] == accumulate
    assert capi.launch_info(m, n, k, STORE)["kernel"] == store


@pytest.mark.parametrize("m,inter,k,fuses", [
    (1, 1040, 1024, 1), (16, 14336, 4096, 1),        # up to 16 tokens always
    (17, 1040, 1024, 0), (24, 7168, 4096, 0),        # owners of up to eight rows
    (28, 7168, 8192, 0),                             # sixteen, up to 32 tokens
    (40, 1040, 1024, 1), (40, 7168, 4096, 1), (48, 3584, 4096, 0), (64, 3584, 4096, 1),
    (17, 14336, 4096, 1), (24, 9488, 256, 1),        # no K split
    (65, 1040, 1024, 1), (1000, 14336, 4096, 1), (17, 1032, 1024, 0), (0, 1040, 1024, 0)])
def test_where_gate_up_takes_swiglu_in(capi, m, inter, k, fuses):
    assert capi.lib.hfrk_gate_up_fuses(m, inter, k, 0) == fuses


def test_a_pinned_projection_is_a_launch_of_its_own_above_16_tokens(capi):
    for m, bucket in ((16, 16), (40, 48), (64, 64), (200, 64)):
        assert capi.lib.hfrk_gate_up_fuses(m, 1040, 1024, 0) == 1
        capi.lib.hfrk_tuning_set(bucket, 2080, 1024, 2, 3)
        try:
            assert capi.lib.hfrk_gate_up_fuses(m, 1040, 1024, 0) == int(m <= 16)
            assert capi.lib.hfrk_gate_up_fuses(m, 1056, 1024, 0) == 1
        finally:
            capi.lib.hfrk_tuning_clear()


@pytest.mark.parametrize("m", [17, 65])
def test_rows_that_a_32_bit_column_cannot_count_stay_on_the_skinny_kernel(capi, m):
    """The last wide tile would end past 2^31 and write in front of its row."""
    assert capi.launch_info(m, 2 ** 31 - 200, 16)["kernel"] == CLUSTER
    assert capi.launch_info(m, 2 ** 31 - 300, 16)["kernel"] == WIDE
    assert capi.lib.hfrk_wide_gemm_fp8(16, 16, 16, 16, 0, m, 2 ** 31 - 200, 16, 16, 0, 0, 1, 0, 0, 0, 0, 0, 0, 0) == 6


@pytest.mark.parametrize("kernel", [CLUSTER, STREAMK])
@pytest.mark.parametrize("m,columns", [(1, 32), (16, 32), (17, 64), (32, 64), (33, 128), (48, 128), (64, 128)])
def test_shared_memory_covers_the_tmem_columns(capi, kernel, m, columns):
    """CTAs of any two kernels that fit on an SM by shared memory fit by TMEM columns (512) too."""
    if kernel == CLUSTER:
        columns = 32 if m <= 32 else 64
    for stages in (2, 3, 8):
        for split in ((1, 4) if kernel == CLUSTER else (0,)):
            info = capi.launch_info(m, 8192, 8192, kernel=kernel, num_stages=stages, split_k=split)
            assert info["num_stages"] == stages and (info["smem_bytes"] + 1024) * 512 >= columns * 228 * 1024

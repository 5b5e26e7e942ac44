"""Lists of host-buffer calls whose results land on other calls' inputs: every input is read before any result."""
import pytest
import torch


@pytest.fixture(scope="module")
def capi(native_build):
    from hf_rocm_kernels import _capi

    return _capi


def _inputs_first(capi, calls):
    """``calls`` = [(A address, D address, accumulate, D_in address or 0)], each 4 x 64 x 128 with 16-bit D."""
    array = (capi.HostCall * len(calls))()
    for slot, (a, d, accumulate, d_in) in zip(array, calls):
        slot.A_host, slot.W_dev, slot.D_host, slot.scale_dev = a, 0x100, d, 0x100
        slot.m, slot.n, slot.k, slot.w_row_stride = 4, 64, 128, 128
        slot.d_dtype, slot.accumulate, slot.D_in_host = 1, accumulate, d_in
    return capi.lib.hfrk_host_batch_inputs_first(array, len(calls))


A, D, SIZE = 0x10000, 0x40000, 512     # both blocks of a call hold 512 bytes


@pytest.mark.parametrize("calls,expect", [
    ([(A, D, 1, 0), (A + SIZE, D + SIZE, 1, 0), (A + 2 * SIZE, D + 2 * SIZE, 1, 0)], 0),     # blocks of their own
    ([(A, D + SIZE, 1, 0), (A, D, 1, 0)], 0),                                               # shared input, any order
    ([(A, D, 1, 0), (A, D, 0, 0)], 0),                                                       # shared result, not read
    ([(A, D, 1, 0), (A, D, 1, 0)], 1),                                                       # shared result, read
    ([(A, D, 1, 0), (A, D + SIZE, 0, 0), (A, D + SIZE - 2, 1, D + 2 * SIZE)], 0),
    ([(A, D, 0, 0), (A, D + SIZE, 1, D + SIZE - 2)], 1),                                     # D_in ends in a result
    ([(A, D, 0, 0), (A, D + 4 * SIZE, 0, 0), (A, D + 2 * SIZE, 1, 0)], 0),                   # between two results
    ([(A, D, 0, 0), (D + SIZE - 1, D + SIZE, 0, 0)], 1),                                     # activations from a result
    ([(A, D, 0, 0), (D + SIZE, D + 4 * SIZE, 0, 0)], 0),                                     # right behind it
    ([(D, D, 0, 0)], 0),                                                                     # a call's own blocks
    ([(D, A, 0, 0), (A + SIZE, D, 0, 0)], 0),                                                # an earlier call's input
])
def test_which_lists_have_their_inputs_read_first(capi, calls, expect):
    assert _inputs_first(capi, calls) == expect


@pytest.mark.gpu
@pytest.mark.parametrize("pinned", [True, False])
@pytest.mark.parametrize("count", [3, 80])          # 80 blocks that cannot be merged: more than the library's ring of events
def test_results_over_inputs_of_later_calls(capi, pinned, count):
    """All calls accumulate into one block and the last one's activations lie in it: each call still sees what
    the block held at first, and the last call's result is what remains."""
    dev = torch.device("cuda:0")
    m, n, k = 16, 8192, 1024
    gen = torch.Generator().manual_seed(count)
    d0 = torch.randn((m, n), generator=gen).bfloat16()
    d_host = d0.clone().pin_memory() if pinned else d0.clone()
    # activation bytes of the last call: the first m * k bytes of the results' block
    d_host.view(torch.uint8).view(-1)[:m * k] = torch.randint(0, 120, (m * k,), generator=gen, dtype=torch.uint8)
    start = d_host.clone()
    scale = torch.tensor([2e-4], device=dev)
    w = torch.randint(0, 120, (n, k), dtype=torch.uint8, generator=gen).view(torch.float8_e4m3fn).to(dev)
    calls = []
    for i in range(count):
        a = torch.randint(0, 120, (m, k + 16), generator=gen, dtype=torch.uint8)
        a = a.pin_memory() if pinned else a
        a = a.view(-1)[:m * k].view(m, k)
        if i == count - 1:
            a = d_host.view(torch.uint8).view(-1)[:m * k].view(m, k)
        calls.append((a.view(torch.float8_e4m3fn), w, d_host, scale, True))
    want = start.to(dev)
    capi.check(capi.skinny_gemm(start.view(torch.uint8).view(-1)[:m * k].view(m, k).view(torch.float8_e4m3fn).to(dev), w, want, scale))
    batch = capi.HostBatch(calls, dev)
    assert capi.lib.hfrk_host_batch_inputs_first(batch.array, count) == 1
    stream = torch.cuda.Stream()
    for _ in range(3):
        d_host.copy_(start)
        capi.check(batch.queue(stream))
        stream.synchronize()
        assert torch.equal(d_host, want.cpu())
    assert capi.device_status(clear=True)[0] == 0


@pytest.mark.gpu
def test_a_batch_that_fails_half_way_is_joined_to_its_stream(capi):
    """The third call's weight pitch is refused after two calls were queued with their copies: one synchronise of
    the stream still covers those, and a batch on the same scratch right behind it is not disturbed."""
    dev = torch.device("cuda:0")
    m, n, k = 16, 28672, 1024                        # every result is a group of its own
    gen = torch.Generator().manual_seed(9)
    scale = torch.tensor([2e-4], device=dev)
    calls, want = [], []
    for i in range(6):
        a = torch.randint(0, 120, (m, k), generator=gen, dtype=torch.uint8)
        w = torch.randint(0, 120, (n, k), generator=gen, dtype=torch.uint8).view(torch.float8_e4m3fn).to(dev)
        d_in = torch.randn((m, n), generator=gen).bfloat16().pin_memory()
        expect = d_in.to(dev)
        capi.check(capi.skinny_gemm(a.view(torch.float8_e4m3fn).to(dev), w, expect, scale))
        want.append(expect.cpu())
        calls.append((a.pin_memory().view(torch.float8_e4m3fn), w, torch.zeros((m, n), dtype=torch.bfloat16).pin_memory(), scale,
                      True, d_in))
    batch = capi.HostBatch(calls, dev)
    stream = torch.cuda.Stream()
    for _ in range(3):
        for call in calls:
            call[2].fill_(0.0)
        batch.array[2].w_row_stride = k + 8
        assert batch.queue(stream) == 7              # HFRK_BAD_ALIGNMENT
        stream.synchronize()
        assert all(torch.equal(calls[i][2], want[i]) for i in range(2))
        assert all(int(calls[i][2].count_nonzero()) == 0 for i in range(2, 6))
        assert batch.queue(stream) == 7
        batch.array[2].w_row_stride = k
        capi.check(batch.queue(stream))
        stream.synchronize()
        assert all(torch.equal(call[2], w) for call, w in zip(calls, want))
    assert capi.device_status(clear=True)[0] == 0

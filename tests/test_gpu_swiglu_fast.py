"""The vector kernel of swiglu against the element-by-element one (accurate expf, IEEE division), byte for byte."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _both(gate_up, scale, fp8):
    from hf_rocm_kernels import swiglu

    s = torch.tensor([scale], device=gate_up.device)
    return [swiglu(gate_up, s, force_scalar=flag, out_dtype=fp8).view(torch.uint8) for flag in (False, True)]


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("fp8", [torch.float8_e4m3fn, torch.float8_e4m3fnuz])
@pytest.mark.parametrize("scale", [1.0, 0.021, 37.0, 3e-5, 1e-30, 4e-39, 1e-45, -0.021, -4e-39, -1e-45])
def test_every_16_bit_gate_value(native_build, dtype, fp8, scale):
    """All 65,536 bit patterns as gates (zeros of both signs, subnormals, infinities, NaNs) times four ups; scales
    of both signs, down to those whose reciprocal overflows. Vectors hold neighbouring patterns, so that slow and fast
    vectors (by their largest gate) both occur."""
    gate = torch.arange(65536, dtype=torch.int32, device="cuda").to(torch.int16).view(dtype).view(8192, 8)
    for up in (1.0, -0.37, 0.0, 250.0):
        fast, exact = _both(torch.cat([gate, torch.full_like(gate, up)], dim=1), scale, fp8)
        assert torch.equal(fast, exact)


# one vector per row; fewer vectors than threads; row steps that wrap; more than one pass of the grid
@pytest.mark.parametrize("rows,hidden", [(1, 8), (70000, 8), (333, 24), (4096, 1000), (7, 28672), (513, 4096), (2048, 6656)])
def test_rows_of_any_length(native_build, rows, hidden):
    gen = torch.Generator(device="cuda").manual_seed(rows + hidden)
    gate_up = (3 * torch.randn((rows, 2 * hidden), generator=gen, device="cuda")).to(torch.bfloat16)
    fast, exact = _both(gate_up, 0.021, torch.float8_e4m3fn)
    assert torch.equal(fast, exact)


def test_no_columns_still_zeroes_the_buffer(native_build):
    from hf_rocm_kernels import swiglu

    buffer = torch.ones((5, 16), dtype=torch.float16, device="cuda")
    out = swiglu(torch.empty((5, 0), dtype=torch.float16, device="cuda"), torch.ones(1, device="cuda"), buffer)
    assert tuple(out.shape) == (5, 0) and int(buffer.count_nonzero()) == 0

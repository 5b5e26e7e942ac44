"""Automatic launch shapes against float64: the GEMM for 17 to 256 tokens per launch with the tokens on the tensor core's M side: plain calls above 64
tokens (and above 16 in more than one wave), the fused gate/up + swiglu call above 16, store mode, and some small shapes of the skinny kernel."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def capi(native_build):
    from hf_rocm_kernels import _capi

    return _capi


@pytest.fixture(scope="module")
def dev():
    return torch.device("cuda:0")


def _ok(capi):
    torch.cuda.synchronize()
    code, word = capi.device_status(clear=True)
    assert code == 0, f"device status word {word:#x}"


def _operands(m, n, k, fp8, dev):
    gen = torch.Generator(device=dev).manual_seed(m * 1009 + n * 31 + k)
    a = torch.randn((m, k), generator=gen, device=dev).to(torch.float8_e4m3fn).view(torch.uint8)
    w = (torch.randn((n, k), generator=gen, device=dev) * 30).to(torch.float8_e4m3fn).view(torch.uint8)
    if fp8 == torch.float8_e4m3fnuz:
        a, w = (torch.where(t == 0x80, torch.zeros_like(t), t) for t in (a, w))
    return a.view(fp8), w.view(fp8), torch.tensor([1.0 / (30.0 * k ** 0.5)], device=dev)


def _bound(ref, a, w, scale, dtype):
    """One step of the output type, and four standard deviations of the fp32 roundings of a random-walk sum."""
    step = {torch.float16: 2.0 ** -10, torch.bfloat16: 2.0 ** -7, torch.float32: 2.0 ** -22}[dtype]
    walk = (a.double().square() @ w.double().square().t()).sqrt() * scale.double().abs()
    return ref.abs() * step + 4 * 2.0 ** -23 * (a.size(1) / 32 + 1) ** 0.5 * walk + (2.0 ** -24 if dtype == torch.float16 else 0)


# one accumulator and two, the edges between them; tiles that end inside the matrix and past it; rows of D
# that are not 16-byte aligned; a K tail; one K block; K splits of two to six; two launches
@pytest.mark.parametrize("m,n,k", [(65, 4096, 4096), (128, 6144, 4096), (129, 6144, 4096), (136, 1001, 1040), (256, 28672, 512),
                                   (255, 4104, 5120), (256, 4096, 14336), (70, 17, 128), (200, 1280, 8192), (130, 33, 16),
                                   (257, 2000, 2064), (513, 1040, 256), (100, 8192, 1024), (30, 39840, 1024),
                                   # up to 16 tokens: K splits down to one K block per CTA (few tiles), and the
                                   # grids that stay two clusters below the device's capacity
                                   (4, 1104, 1104), (16, 1808, 1808), (3, 17, 256), (11, 10336, 6992)])
@pytest.mark.parametrize("fp8,dtype", [(torch.float8_e4m3fn, torch.bfloat16), (torch.float8_e4m3fnuz, torch.float16)])
def test_wide_gemm_against_float64(capi, dev, m, n, k, fp8, dtype):
    a, w, scale = _operands(m, n, k, fp8, dev)
    gen = torch.Generator(device=dev).manual_seed(5)
    d_in = torch.randn((m, n), generator=gen, device=dev).to(dtype)
    backing = torch.full((m * n + 64,), 9.0, dtype=dtype, device=dev)
    d = backing[32:32 + m * n].view(m, n)
    prod = (a.double() @ w.double().t()) * scale.double()
    for start, ref in ((d_in, prod + d_in.double()), (torch.zeros_like(d_in), prod)):
        d.copy_(start)
        capi.check(capi.skinny_gemm(a, w, d, scale))
        _ok(capi)
        assert bool(((d.double() - ref).abs() <= _bound(ref, a, w, scale, dtype)).all())
    first = d.clone()
    for _ in range(2):                       # store mode: what D held before does not matter; same bits every time
        d.fill_(float("nan"))
        torch.ops._HFRK_C.skinny_gemm_store(a, w.t(), d, scale)
        _ok(capi)
        assert torch.equal(d, first)
    assert bool((backing[:32] == 9).all() and (backing[-32:] == 9).all())


def test_wide_gemm_float32_output_and_padded_weights(capi, dev):
    m, n, k = 150, 1000, 2048
    a, w, scale = _operands(m, n, k, torch.float8_e4m3fn, dev)
    padded = torch.zeros((n, k + 48), dtype=torch.uint8, device=dev)
    padded[:, :k] = w.view(torch.uint8)
    wp = padded.view(torch.float8_e4m3fn)[:, :k]
    d = torch.ones((m, n), dtype=torch.float32, device=dev)
    capi.check(capi.skinny_gemm(a, wp, d, scale))
    _ok(capi)
    ref = (a.double() @ w.double().t()) * scale.double() + 1.0
    assert bool(((d.double() - ref).abs() <= _bound(ref, a, w, scale, torch.float32)).all())


@pytest.mark.parametrize("m,inter,k", [(17, 1040, 256), (64, 3584, 8192), (128, 14336, 4096), (129, 2048, 4096), (200, 3584, 8192),
                                       (256, 28672, 512), (300, 1040, 512), (33, 16, 128), (96, 48, 16)])
@pytest.mark.parametrize("act,fp8", [(torch.bfloat16, torch.float8_e4m3fn), (torch.float16, torch.float8_e4m3fnuz)])
def test_wide_gate_up_swiglu_against_the_two_launches(capi, dev, m, inter, k, act, fp8):
    """The same fp8 values as GEMM + swiglu except where another order of the fp32 sum moves the 16-bit
    projection across a rounding boundary and that moves the result across one of fp8. A sum over K / 32
    steps in another order changes by less than 2^-21 of a typical projection, which crosses a 16-bit
    boundary (2^-8 apart at the coarsest) for at most one value in 2^13 and then moves the product by one
    16-bit step, across an fp8 boundary (2^-4 apart) in one of 2^4 (bf16) such cases: 2^-17 each for gate and
    up. Twice that and a margin of eight values for small cases."""
    from hf_rocm_kernels import skinny_gemm, swiglu

    a, w, scale = _operands(m, 2 * inter, k, fp8, dev)
    act_scale = torch.tensor([0.02], device=dev)
    gate_up = torch.zeros((m, 2 * inter), dtype=act, device=dev)
    skinny_gemm(a, w.t(), scale, gate_up)
    expect = swiglu(gate_up, act_scale, out_dtype=fp8)
    backing = torch.full((m * inter + 64,), 0x55, dtype=torch.uint8, device=dev)
    out = backing[32:32 + m * inter].view(m, inter).view(fp8)
    zeroed = torch.ones((m, 24), dtype=act, device=dev)
    torch.ops._HFRK_C.gate_up_swiglu(a, w.t(), out, scale, act_scale, zeroed, act == torch.bfloat16)
    _ok(capi)
    differ = int((out.view(torch.uint8) != expect.view(torch.uint8)).sum())
    assert differ <= 8 + out.numel() * 2.0 ** -15, differ
    step = (out.float() - expect.float()).abs()
    assert bool((step <= expect.float().abs() * 2.0 ** -3 + 2.0 ** -9).all())    # one fp8 step
    assert int(zeroed.count_nonzero()) == 0
    assert bool((backing[:32] == 0x55).all() and (backing[-32:] == 0x55).all())


def test_explicit_launch_shapes_stay_on_the_skinny_kernel(capi, dev):
    """A requested split or a tuned token bucket means the 64-token launches it was made for."""
    a, w, scale = _operands(130, 2000, 4096, torch.float8_e4m3fn, dev)
    ref = (a.double() @ w.double().t()) * scale.double()
    outs = []
    for kw in ({"split_k": 3}, {"variant": 1}):
        d = torch.zeros((130, 2000), dtype=torch.bfloat16, device=dev)
        capi.check(capi.skinny_gemm_ex(a, w, d, scale, **kw))
        outs.append(d)
    capi.lib.hfrk_tuning_set(64, 2000, 4096, 2, 3)
    try:
        d = torch.zeros((130, 2000), dtype=torch.bfloat16, device=dev)
        capi.check(capi.skinny_gemm(a, w, d, scale))
        outs.append(d)
    finally:
        capi.lib.hfrk_tuning_clear()
    _ok(capi)
    for d in outs:
        assert bool(((d.double() - ref).abs() <= _bound(ref, a, w, scale, torch.bfloat16)).all())


@pytest.mark.parametrize("tokens", [17, 100, 256])
@pytest.mark.parametrize("inter", [1040, 1032])            # rows that split into 16-byte pieces, and rows that do not
def test_mlp_chain_above_16_tokens(capi, dev, tokens, inter):
    """The chain against itself with swiglu as a launch of its own, eager and from a graph."""
    from hf_rocm_kernels.combined_ops import llama_mlp_combined_ops

    hidden = 1024
    gen = torch.Generator(device=dev).manual_seed(3)
    attn, residual = (torch.randn((tokens, hidden), generator=gen, device=dev).to(torch.bfloat16) for _ in range(2))
    _, w_gu, s_gu = _operands(1, 2 * inter, hidden, torch.float8_e4m3fn, dev)
    w_dn = (torch.randn((hidden, (inter + 15) // 16 * 16), generator=gen, device=dev) * 30).to(torch.float8_e4m3fn)[:, :inter]
    s_dn = torch.tensor([0.02 / (30.0 * inter ** 0.5)], device=dev)
    one, act_scale = torch.tensor([0.02], device=dev), torch.tensor([0.02], device=dev)
    norm = torch.ones(hidden, dtype=torch.bfloat16, device=dev)

    def chain(res, **kw):
        return llama_mlp_combined_ops(attn, res, norm, 1e-5, w_gu.t(), one, s_gu * 0.02, w_dn.t(), act_scale, s_dn, **kw)

    if inter % 16:
        with pytest.raises(RuntimeError):                  # the down projection's K
            chain(residual.clone())
        return
    out, res = chain(residual.clone())
    parts, res_parts = chain(residual.clone(), fuse_swiglu=False)
    with pytest.raises(RuntimeError):
        chain(residual.clone(), fuse_swiglu=True)
    _ok(capi)
    assert torch.equal(res, res_parts)
    error = (out.double() - parts.double()).norm() / parts.double().norm()
    assert float(error) <= 2.0 ** -9                       # a few outputs one bf16 step (2^-8) apart at most
    static, side = residual.clone(), torch.cuda.Stream(dev)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.stream(side):
        torch.cuda.synchronize()
        with torch.cuda.graph(graph, stream=side):
            g_out, _ = chain(static)
    static.copy_(residual)
    graph.replay()
    _ok(capi)
    assert torch.equal(g_out, out)


@pytest.mark.parametrize("act,fp8", [(torch.bfloat16, torch.float8_e4m3fn), (torch.float16, torch.float8_e4m3fnuz)])
@pytest.mark.parametrize("scale", [0.02, -0.02, 4e-39, -4e-39, 1e-45, -1e-45])
def test_fused_swiglu_under_extreme_scales(capi, dev, act, fp8, scale):
    """One K block, so that the projection is the same sum in both forms: the same bytes, zero rows (a projection
    of zero times a scale whose double overflows) among them."""
    from hf_rocm_kernels import skinny_gemm, swiglu

    m, inter, k = 40, 64, 128
    a, w, s = _operands(m, 2 * inter, k, fp8, dev)
    a.view(torch.uint8)[::3] = 0
    act_scale = torch.tensor([scale], device=dev)
    gate_up = torch.zeros((m, 2 * inter), dtype=act, device=dev)
    skinny_gemm(a, w.t(), s, gate_up)
    expect = swiglu(gate_up, act_scale, out_dtype=fp8, force_scalar=True)
    out = torch.empty((m, inter), dtype=fp8, device=dev)
    none = torch.empty((m, 0), dtype=act, device=dev)
    torch.ops._HFRK_C.gate_up_swiglu(a, w.t(), out, s, act_scale, none, act == torch.bfloat16)
    _ok(capi)
    assert torch.equal(out.view(torch.uint8), expect.view(torch.uint8))


def _shapes(capi, m, n, k, split, swiglu):
    """Launch shapes with this K split: one and two CTAs per SM, two stages and as many as fit, of the tile heights
    that the device holds the lowest, the highest and the ones whose column groups do not divide by the split."""
    step = 32 if swiglu else 16
    shapes = []
    for per_sm in (1, 2):
        for stages in (2, 0):
            fits = []
            for tile in range(32, 257, step):
                out = (capi.ctypes.c_int * 8)()
                if capi.lib.hfrk_gemm_launch_info(m, n, k, 2 * swiglu, 3, split, tile, stages, per_sm, out) == 0:
                    fits.append(tile)
            uneven = [t for t in fits if t // step % split]
            shapes += [(per_sm, stages, t) for t in sorted({*fits[:1], *uneven[:1], *uneven[-1:], *fits[-1:]})]
    return shapes


@pytest.mark.parametrize("split", range(1, 9))
@pytest.mark.parametrize("m", [40, 128, 200])              # one accumulator, all its rows, two
@pytest.mark.parametrize("n,dtype", [(1000, torch.bfloat16), (1002, torch.float16), (1003, torch.bfloat16), (1003, torch.float32)])
def test_pinned_launch_shapes_against_float64(capi, dev, m, n, dtype, split):
    """Rows of D that are 16-byte aligned, 4-byte aligned and neither; accumulating and storing; N that ends
    inside a tile; eleven K blocks, the last one short, shared out unevenly."""
    k = 1296
    a, w, scale = _operands(m, n, k, torch.float8_e4m3fn, dev)
    d_in = torch.randn((m, n), generator=torch.Generator(device=dev).manual_seed(5), device=dev).to(dtype)
    prod = (a.double() @ w.double().t()) * scale.double()
    bound, bound_in = _bound(prod, a, w, scale, dtype), _bound(prod + d_in.double(), a, w, scale, dtype)
    shapes = _shapes(capi, m, n, k, split, False)
    assert shapes and (m > 40 or {s[:2] for s in shapes} == {(1, 0), (1, 2), (2, 0), (2, 2)})
    for per_sm, stages, tile in shapes:
        backing = torch.full((m * n + 64,), 9.0, dtype=dtype, device=dev)
        d = backing[32:32 + m * n].view(m, n)
        pins = dict(split_k=split, tile_rows=tile, num_stages=stages, ctas_per_sm=per_sm)
        d.copy_(d_in)
        capi.check(capi.wide_gemm(a, w, d, scale, **pins))
        _ok(capi)
        assert bool(((d.double() - prod - d_in.double()).abs() <= bound_in).all()), pins
        d.fill_(float("nan"))
        capi.check(capi.wide_gemm(a, w, d, scale, accumulate=False, **pins))
        _ok(capi)
        assert bool(((d.double() - prod).abs() <= bound).all()), pins
        assert bool((backing[:32] == 9).all() and (backing[-32:] == 9).all()), pins


@pytest.mark.parametrize("split", range(1, 9))
@pytest.mark.parametrize("m", [3, 40, 128, 200])
@pytest.mark.parametrize("act,fp8", [(torch.bfloat16, torch.float8_e4m3fn), (torch.float16, torch.float8_e4m3fnuz)])
def test_pinned_swiglu_launch_shapes(capi, dev, m, act, fp8, split):
    """As :func:`test_wide_gate_up_swiglu_against_the_two_launches`, by pinned shapes."""
    from hf_rocm_kernels import skinny_gemm, swiglu

    inter, k = 528, 1296
    a, w, scale = _operands(m, 2 * inter, k, fp8, dev)
    act_scale = torch.tensor([0.02], device=dev)
    gate_up = torch.zeros((m, 2 * inter), dtype=act, device=dev)
    skinny_gemm(a, w.t(), scale, gate_up)
    expect = swiglu(gate_up, act_scale, out_dtype=fp8)
    shapes = _shapes(capi, m, 2 * inter, k, split, True)
    assert shapes or (m == 200 and split > 6)     # no room for the partials of so many
    for per_sm, stages, tile in shapes:
        pins = dict(split_k=split, tile_rows=tile, num_stages=stages, ctas_per_sm=per_sm)
        backing = torch.full((m * inter + 64,), 0x55, dtype=torch.uint8, device=dev)
        out = backing[32:32 + m * inter].view(m, inter).view(fp8)
        capi.check(capi.wide_gemm(a, w, out, scale, act_scale, mid_dtype=act, **pins))
        _ok(capi)
        assert int((out.view(torch.uint8) != expect.view(torch.uint8)).sum()) <= 8 + out.numel() * 2.0 ** -15, pins
        step = (out.float() - expect.float()).abs()
        assert bool((step <= expect.float().abs() * 2.0 ** -3 + 2.0 ** -9).all()), pins
        assert bool((backing[:32] == 0x55).all() and (backing[-32:] == 0x55).all()), pins


# (24, 9488, 256): one launch without a K split; (40, 1040, 1024) with one; (24, 1040, 1024), (48, 3584, 4096): two
@pytest.mark.parametrize("m,inter,k,fuses", [(24, 9488, 256, 1), (40, 1040, 1024, 1), (24, 1040, 1024, 0), (48, 3584, 4096, 0)])
@pytest.mark.parametrize("act,fp8", [(torch.bfloat16, torch.float8_e4m3fn), (torch.float16, torch.float8_e4m3fnuz)])
def test_gate_up_op_runs_what_the_rule_names(capi, dev, m, inter, k, fuses, act, fp8):
    """The bytes of the op are those of the one launch or of the two, also with a launch shape pinned for the
    projection and with a buffer that is no multiple of 16 bytes (two launches in both cases)."""
    from hf_rocm_kernels import swiglu

    a, w, scale = _operands(m, 2 * inter, k, fp8, dev)
    act_scale = torch.tensor([0.02], device=dev)

    def op(cols):
        out, buffer = torch.empty((m, inter), dtype=fp8, device=dev), torch.ones((m, cols), dtype=act, device=dev)
        torch.ops._HFRK_C.gate_up_swiglu(a, w.t(), out, scale, act_scale, buffer, act == torch.bfloat16)
        _ok(capi)
        assert int(buffer.count_nonzero()) == 0
        return out.view(torch.uint8)

    def two_launches():
        gate_up = torch.empty((m, 2 * inter), dtype=act, device=dev)
        torch.ops._HFRK_C.skinny_gemm_store(a, w.t(), gate_up, scale)
        return swiglu(gate_up, act_scale, out_dtype=fp8).view(torch.uint8)

    one = torch.empty((m, inter), dtype=fp8, device=dev)
    capi.check(capi.wide_gemm(a, w, one, scale, act_scale, mid_dtype=act))
    with torch.cuda.device(dev):
        assert capi.lib.hfrk_gate_up_fuses(m, inter, k, 0) == fuses
    assert torch.equal(op(8), one.view(torch.uint8) if fuses else two_launches())
    assert torch.equal(op(5), two_launches() if m * 5 % 8 else op(8))
    capi.lib.hfrk_tuning_set(m, 2 * inter, k, 2, 2)
    try:
        assert torch.equal(op(8), two_launches())
    finally:
        capi.lib.hfrk_tuning_clear()


@pytest.mark.parametrize("tokens,hidden,inter", [(24, 256, 9488), (40, 1024, 1040)])
def test_mlp_block_takes_swiglu_in(capi, dev, tokens, hidden, inter):
    """The block's automatic form above 16 tokens, on shapes where that is one launch, against the two."""
    from hf_rocm_kernels.combined_ops import llama_mlp_combined_ops

    assert capi.lib.hfrk_gate_up_fuses(tokens, inter, hidden, 0) == 1
    gen = torch.Generator(device=dev).manual_seed(3)
    attn, residual = (torch.randn((tokens, hidden), generator=gen, device=dev).to(torch.bfloat16) for _ in range(2))
    _, w_gu, s_gu = _operands(1, 2 * inter, hidden, torch.float8_e4m3fn, dev)
    _, w_dn, s_dn = _operands(2, hidden, inter, torch.float8_e4m3fn, dev)
    act_scale, norm = torch.tensor([0.02], device=dev), torch.ones(hidden, dtype=torch.bfloat16, device=dev)
    outs = [llama_mlp_combined_ops(attn, residual.clone(), norm, 1e-5, w_gu.t(), act_scale, s_gu * 0.02, w_dn.t(), act_scale,
                                   s_dn * 0.02, **kw) for kw in ({}, {"fuse_swiglu": False})]
    _ok(capi)
    assert torch.equal(outs[0][1], outs[1][1])
    error = (outs[0][0].double() - outs[1][0].double()).norm() / outs[1][0].double().norm()
    assert float(error) <= 2.0 ** -9                       # a few outputs one bf16 step (2^-8) apart at most

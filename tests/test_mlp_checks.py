"""What the MLP block refuses before it launches anything: tensors on another device above all (a host
pointer in a kernel is a fault). CPU: fake CUDA tensors through the block. GPU: the op's own check."""
import pytest
import torch
from torch._subclasses.fake_tensor import FakeTensorMode

FP8 = torch.float8_e4m3fn


def _block(tokens, hidden, inter, **other):
    """One call of the block on tensors of device ``cuda``; ``other`` replaces arguments by name."""
    from hf_rocm_kernels.combined_ops import llama_mlp_combined_ops

    def empty(*shape, dtype=FP8, device="cuda"):
        return torch.empty(shape, dtype=dtype, device=device)

    def scale():
        return empty(1, dtype=torch.float32)

    args = {"attn_output": empty(tokens, hidden, dtype=torch.bfloat16), "residual": empty(tokens, hidden, dtype=torch.bfloat16),
            "rms_weight": empty(hidden, dtype=torch.bfloat16), "gate_up_weight": empty(2 * inter, hidden).t(),
            "gate_up_input_scale": scale(), "gate_up_output_scale": scale(), "down_weight": empty(hidden, inter).t(),
            "down_input_scale": scale(), "down_output_scale": scale()}
    args.update((name, make(empty)) for name, make in other.items())
    return llama_mlp_combined_ops(rms_epsilon=1e-5, **args)


# 17 tokens: one launch for gate/up and swiglu from 20 million weights on, two below; 33 tokens: always one
@pytest.mark.parametrize("tokens,hidden,inter", [(17, 4096, 4096), (17, 1024, 1024), (33, 1024, 1024), (256, 1024, 1024)])
@pytest.mark.parametrize("name,make", [
    ("gate_up_output_scale", lambda e: e(1, dtype=torch.float32, device="cpu")),
    ("down_input_scale", lambda e: e(1, dtype=torch.float32, device="cpu")),
    ("down_output_scale", lambda e: e(1, dtype=torch.float32, device="cpu")),
    ("gate_up_output_scale", lambda e: e(2, dtype=torch.float32)),
    ("gate_up_output_scale", lambda e: e(1, dtype=torch.float64)),
    ("down_input_scale", lambda e: e(2, dtype=torch.float32)),
])
def test_block_above_16_tokens_refuses_bad_scales(native_build, tokens, hidden, inter, name, make):
    with FakeTensorMode():
        with pytest.raises(AssertionError):
            _block(tokens, hidden, inter, **{name: make})


@pytest.mark.parametrize("tokens,hidden,inter", [(17, 4096, 4096), (17, 1024, 1024), (33, 1024, 1024)])
def test_block_above_16_tokens_refuses_bad_weights(native_build, tokens, hidden, inter):
    with FakeTensorMode():
        for make in (lambda e: e(2 * inter, hidden, device="cpu").t(), lambda e: e(hidden, 2 * inter), lambda e: e(2 * inter + 1, hidden).t()):
            with pytest.raises(AssertionError):
                _block(tokens, hidden, inter, gate_up_weight=make)
        _block(tokens, hidden, inter)


@pytest.mark.gpu
@pytest.mark.parametrize("tokens", [4, 17])
@pytest.mark.parametrize("position", range(6))
def test_fused_ops_refuse_tensors_of_another_device(native_build, tokens, position):
    """Raised by the host side of the op; nothing is launched."""
    inter, hidden = 32, 64
    tensors = [torch.zeros((tokens, hidden), device="cuda").to(FP8), torch.zeros((2 * inter, hidden), device="cuda").to(FP8).t(),
               torch.zeros((tokens, inter), device="cuda").to(FP8), torch.ones(1, device="cuda"), torch.ones(1, device="cuda"),
               torch.ones((tokens, 8), device="cuda", dtype=torch.bfloat16)]
    ops = [torch.ops._HFRK_C.gate_up_swiglu] + ([torch.ops._HFRK_C.skinny_gemm_swiglu] if tokens <= 16 else [])
    for op in ops:
        op(*tensors, True)                                    # all on the GPU: runs
        torch.cuda.synchronize()
        # cpu() of a transposed tensor keeps its strides
        mixed = [t.cpu() if i == position else t for i, t in enumerate(tensors)]
        with pytest.raises(RuntimeError, match="on one GPU"):
            op(*mixed, True)

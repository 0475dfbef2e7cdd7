"""Operands that a product must refuse before their addresses reach a kernel."""
import pytest
import torch


class _OnDevice:
    """What ``linear_xielu`` asks of its parameters, answered as a tensor on the device would."""
    is_cuda, dtype = True, torch.float32
    numel, is_contiguous = staticmethod(lambda: 2), staticmethod(lambda: True)


@pytest.mark.parametrize("rows", [1, 129, 300, 1024, 1025])
@pytest.mark.parametrize("params", [_OnDevice(), torch.zeros(2)])
def test_xielu_of_host_operands_is_refused(rows, params, monkeypatch):
    from dispec_b200.ops import gemm, library
    launched = []
    for kernel in ("_pairs", "_stream", "_tcgen05", "_simt", "_split", "_library"):
        monkeypatch.setattr(gemm, kernel, lambda *a, **k: launched.append(a))
    x, w = torch.zeros(rows, 64, dtype=torch.bfloat16), torch.zeros(32, 64, dtype=torch.bfloat16)
    with pytest.raises(library.KernelError, match="CUDA tensors only"):
        gemm.linear_xielu(x, w, params)
    assert not launched

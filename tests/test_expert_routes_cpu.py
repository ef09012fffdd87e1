"""Which kernels an expert layer calls, without a GPU: the library is a recorder."""
import types

import pytest
import torch

from atlas_b200.layers.moe import ExpertWeights
from atlas_b200.ops import cuda_ext


class _Recorder:
    def __init__(self):
        self.calls = []

    def __getattr__(self, name):
        return lambda *a: self.calls.append((name, a)) or 0


@pytest.fixture
def calls(monkeypatch):
    lib = _Recorder()
    fake = types.SimpleNamespace(lib=lambda: lib, _stream=lambda: 0, _num_sms={0: 148}, _status_ptr={0: 0}, _dev=lambda t: 0,
                                 _ptr=lambda t: None if t is None else t.data_ptr(), _check=lambda rc, what: None,
                                 checked=types.SimpleNamespace(ENABLED=False), KernelError=RuntimeError, relu_squared=lambda t: t)
    monkeypatch.setattr(cuda_ext, "K", fake)
    return lib.calls


def _run(T, E, H, I, experts, activation, dtype=torch.bfloat16):
    ids = torch.arange(T * 2, dtype=torch.int32).view(T, 2) % E
    unit = (7.0, 1.702, 1.0) if activation == "clamped_glu" else None
    return cuda_ext._moe_local(torch.zeros(T, H, dtype=dtype), torch.ones(T, 2), ids, experts, 0, activation=activation, unit=unit)


@pytest.mark.parametrize("activation", ["relu2", "clamped_glu"])
@pytest.mark.parametrize("dtype,H,I", [(torch.float32, 64, 64), (torch.bfloat16, 72, 64), (torch.bfloat16, 64, 40)])
def test_experts_in_fp32_sums(calls, dtype, H, I, activation):
    """fp32 experts, and bf16 ones of widths that the tensor-core tiles do not take, go through the plain kernels: row lists without
    pairs of tiles, the two products, the weighted sum."""
    n1 = I if activation == "relu2" else 2 * I
    ex = ExpertWeights("dense", torch.zeros(4, n1, H, dtype=dtype), torch.zeros(4, H, I, dtype=dtype))
    out = _run(5, 4, H, I, ex, activation, dtype)
    assert out.shape == (5, H) and out.dtype == dtype
    assert [c[0] for c in calls] == ["atlas_moe_align", "atlas_moe_plain_gemm", "atlas_moe_plain_gemm", "atlas_moe_plain_combine"]
    assert calls[0][1][9] is None


@pytest.mark.parametrize("kind", ["dense", "fp8_block", "nvfp4"])
def test_only_nvfp4_products_get_pairs_of_tiles(calls, kind):
    ex = ExpertWeights.from_dense(torch.randn(2, 512, 256).bfloat16(), torch.randn(2, 256, 256).bfloat16(), kind)
    _run(40, 2, 256, 256, ex, "silu_glu")
    assert calls[0][0] == "atlas_moe_align" and (calls[0][1][9] is not None) == (kind == "nvfp4")

"""Host-side behaviour of the Python API that needs no GPU."""
import pytest
import torch

import flash_colreduce_b200 as fc
from oracle import oracle_colreduce, oracle_valid_scores


def test_exports_match_the_reference_package():
    for name in ("flash_colreduce", "naive_colreduce", "__version__"):
        assert hasattr(fc, name)


def test_cpu_tensors_are_rejected_like_the_reference():
    q = torch.zeros(1, 1, 4, 8, dtype=torch.float16)
    with pytest.raises(ValueError, match="Query and key tensors must be on CUDA device."):
        fc.flash_colreduce(q, q, "sum")


def test_no_cpu_fallback_exists():
    import inspect

    from flash_colreduce_b200 import op

    src = inspect.getsource(op)
    assert "oracle" not in src and "naive_colreduce" not in src


@pytest.mark.parametrize("m,n", [(5, 5), (4, 9), (9, 4), (128, 1024)])
def test_valid_scores(m, n):
    assert fc.valid_scores(2, 3, m, n, True) == oracle_valid_scores(2, 3, m, n, True)
    assert fc.valid_scores(2, 3, m, n, False) == 6 * m * n


@pytest.mark.parametrize("red", ["sum", "mean", "max"])
@pytest.mark.parametrize("causal", [False, True])
def test_dense_definition_matches_oracle(red, causal):
    g = torch.Generator().manual_seed(2)
    q = torch.randn(2, 2, 37, 8, generator=g)
    k = torch.randn(2, 2, 53, 8, generator=g)
    got = fc.naive_colreduce(q, k, red, causal, block_rows=10)
    torch.testing.assert_close(got, oracle_colreduce(q, k, red, causal), rtol=1e-5, atol=1e-7)
    with pytest.raises(ValueError, match="Invalid reduction"):
        fc.naive_colreduce(q, k, "prod")


def test_signature_is_the_reference_operator_signature():
    """flash_colreduce(query, key, reduction, is_causal=False, scale=None), flash_colreduce/flash.py:311-317."""
    import inspect

    params = inspect.signature(fc.flash_colreduce).parameters
    assert list(params) == ["query", "key", "reduction", "is_causal", "scale"]
    assert params["is_causal"].default is False and params["scale"].default is None
    assert all(p.kind is inspect.Parameter.POSITIONAL_OR_KEYWORD for p in params.values())
    naive = inspect.signature(fc.naive_colreduce).parameters
    assert list(naive)[:5] == ["query", "key", "reduction", "is_causal", "scale"]  # naive.py:8-14


@pytest.mark.parametrize("dtype", [torch.float16, torch.float32])
def test_operands_tma_cannot_describe_are_copied(dtype):
    """An unaligned base, a transposed inner dimension, rows of odd width, a head dimension that is no multiple of 16 bytes:
    what goes in has the values, unit inner stride, strides of whole 16 bytes and an aligned base."""
    from flash_colreduce_b200.op import _tma_ready

    unit = 16 // torch.empty(0, dtype=dtype).element_size()
    x = torch.randn(2, 3, 5, 16).to(dtype)
    shifted = torch.empty(x.numel() + 1, dtype=dtype)[1:].view_as(x).copy_(x)
    assert shifted.is_contiguous() and shifted.data_ptr() % 16 != 0
    inner = x.transpose(2, 3).contiguous().transpose(2, 3)
    wide = torch.zeros(2, 3, 5, 17, dtype=dtype)[..., :16].copy_(x)
    for y in (shifted, inner, wide, x[..., :13]):
        z = _tma_ready(y)
        assert torch.equal(z[..., :y.shape[-1]], y) and not z[..., y.shape[-1]:].any()
        assert z.data_ptr() % 16 == 0 and z.stride(3) == 1 and z.shape[-1] % unit == 0
        assert all(z.stride(i) % unit == 0 for i in range(3))
    assert _tma_ready(x) is x
    bmhd = torch.randn(2, 5, 3, 16).to(dtype).transpose(1, 2)
    assert _tma_ready(bmhd) is bmhd

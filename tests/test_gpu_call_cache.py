"""Repeated call signatures skip validation and planning (needs a B200): what the skipped checks stood for still holds.

The cache key has shapes, strides, types, devices and options, no addresses: a view that starts at another alignment has the
signature of an aligned one, and each element of the key stands between a cached plan and a call that it does not fit.
"""
import pytest
import torch

from conftest import assert_parity
from oracle import oracle_colreduce

pytestmark = pytest.mark.gpu

B, H, M, N, D = 2, 3, 96, 200, 64


def _tensor(rows, seed, dtype=torch.float16, offset=0, layout="bhmd"):
    """CPU values and a CUDA tensor of them whose storage starts `offset` elements after an allocation."""
    g = torch.Generator().manual_seed(seed)
    x = torch.randn(B, H, rows, D, generator=g).to(dtype)
    buf = torch.empty(x.numel() + offset, dtype=dtype, device="cuda:0")[offset:]
    if layout == "bhmd":
        dev = buf.view(B, H, rows, D)
    else:
        dev = buf.view(B, rows, H, D).transpose(1, 2)
    dev.copy_(x)
    return x, dev


def _check(q, k, red="sum", causal=True, scale=None):
    from flash_colreduce_b200 import flash_colreduce

    got = flash_colreduce(q[1], k[1], red, is_causal=causal, scale=scale)
    extra = {torch.float16: 2.0 ** -11, torch.bfloat16: 2.0 ** -8, torch.float32: 2.0 ** -11}[q[0].dtype]
    assert_parity(got, oracle_colreduce(q[0], k[0], red, causal, scale=scale), red, extra_rtol=extra)


def test_an_unaligned_view_of_a_cached_signature():
    q, k = _tensor(M, 1), _tensor(N, 2)
    _check(q, k)
    _check(q, k)
    for q_off, k_off in ((1, 0), (0, 1), (3, 5), (0, 0), (8, 8)):  # elements of two bytes; 8 are 16 bytes again
        qo, ko = _tensor(M, 3 + q_off, offset=q_off), _tensor(N, 20 + k_off, offset=k_off)
        assert qo[1].stride() == q[1].stride() and (qo[1].data_ptr() % 16 == 0) == (q_off % 8 == 0)
        _check(qo, ko)


def test_one_element_of_the_signature_changed_at_a_time():
    q, k = _tensor(M, 1), _tensor(N, 2)
    base = dict(red="sum", causal=True, scale=None)
    variants = [dict(red="max"), dict(red="mean"), dict(causal=False), dict(scale=0.3), dict(scale=-0.3)]
    for _ in range(2):  # the second time every signature is in the cache
        _check(q, k, **base)
        for v in variants:
            _check(q, k, **{**base, **v})
        _check(_tensor(M, 4, layout="bmhd"), k)
        _check(q, _tensor(N, 5, layout="bmhd"))
        _check(_tensor(M + 1, 6), k)
        _check(q, _tensor(N - 1, 7))
        _check(_tensor(M, 8, torch.bfloat16), _tensor(N, 9, torch.bfloat16))


def test_a_repeated_signature_is_planned_once(monkeypatch):
    from flash_colreduce_b200 import flash_colreduce, op

    monkeypatch.setattr(op, "_CALL_CACHE", {})
    q, k = _tensor(M, 1), _tensor(N, 2)
    want = flash_colreduce(q[1], k[1], "sum", is_causal=True)
    assert len(op._CALL_CACHE) == 1
    flash_colreduce(_tensor(M, 3, offset=1)[1], k[1], "max")  # a copy goes in: nothing to keep
    assert len(op._CALL_CACHE) == 1

    def never(*args):
        raise AssertionError("planned again")

    monkeypatch.setattr(op, "_prepare", never)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        again = flash_colreduce(q[1], k[1], "sum", is_causal=True)
    torch.cuda.current_stream().wait_stream(side)
    assert torch.equal(want, again)
    for bad in (dict(query=q[1].cpu()), dict(key=k[1][:, :2]), dict(reduction="median"), dict(key=k[1].float())):
        with pytest.raises((ValueError, TypeError)):
            flash_colreduce(**{**dict(query=q[1], key=k[1], reduction="sum", is_causal=True), **bad})

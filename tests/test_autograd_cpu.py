"""The autograd functions of ops/autograd.py on the CPU path."""
import pytest
import torch

from hetu_galvatron_b200.ops import autograd as A


@pytest.mark.parametrize("layout", ["rows apart", "columns first"])
def test_packed_attention_under_saved_tensor_hooks(layout):
    """A hook may hand the packed projection back in other strides than it was saved with."""
    torch.manual_seed(0)
    b, s, hq, hk, dh = 2, 5, 4, 2, 8
    cfg = A.AttnCfg(batch=b, hq=hq, hk=hk, dh=dh, causal=True)
    x = torch.randn(s * b, (hq + 2 * hk) * dh, requires_grad=True)
    do = torch.randn(s * b, hq * dh)
    want, = torch.autograd.grad(A.packed_attention(x * 1.0, cfg), x, do)

    def unpack(t):
        if t is None or t.dim() != 2:
            return t
        if layout == "columns first":
            return t.t().contiguous().t()
        return torch.cat([t, torch.zeros(t.shape[0], 8, dtype=t.dtype)], 1)[:, :t.shape[1]]

    with torch.autograd.graph.saved_tensors_hooks(lambda t: t, unpack):
        o = A.packed_attention(x * 1.0, cfg)
    got, = torch.autograd.grad(o, x, do)
    assert torch.equal(got, want)

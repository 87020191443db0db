"""The autograd functions of ops/autograd.py and the gradient norm over their buffers, on the CPU path."""
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


def test_gradient_norm_keeps_the_bits_of_small_buckets():
    """Each bucket's squares are summed on their own: 64 buckets of norm one beside one of norm 4096 are not rounded away one by
    one (fp32 resolves 2 at 4096^2)."""
    from hetu_galvatron_b200.parallel.zero import ParamBucket, ZeroEngine
    engine = ZeroEngine()
    for i in range(65):
        b = engine.add_bucket(ParamBucket("b%d" % i, [torch.nn.Parameter(torch.zeros(4))], None))
        b._ensure_grad()
        b.grad_flat[0] = 4096.0 if i == 0 else 1.0
        b.grad_shard = b.grad_flat
    exact = (4096.0 ** 2 + 64) ** 0.5
    assert abs(engine.grad_norm().item() - exact) < 2.0 ** -23 * 2 * exact

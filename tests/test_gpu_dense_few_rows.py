"""Few-row products around the lines where they change kernel, tile width and k-blocks per stage, against fp32."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def _rand(*shape, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn(*shape, generator=g, device="cuda").bfloat16()


@pytest.mark.parametrize("m", [2, 3, 4, 5, 8, 9, 63, 64, 65, 128, 129])
@pytest.mark.parametrize("k", [72, 320, 1096])
@pytest.mark.parametrize("plain,pairs", [(1024, 0), (1056, 0), (3040, 544), (4128, 4096), (17, 9600)])
def test_projection(m, k, plain, pairs):
    from flashrec_b200.lm_layers import MergedProjection, interleave_rows

    a, w = _rand(m, k, seed=m), _rand(plain, k, seed=1) * k ** -0.5
    proj = MergedProjection(k)
    proj.add("store_f32", w)
    outs = [torch.full((m, plain), float("nan"), device="cuda")]
    if pairs:
        gate, up = _rand(pairs, k, seed=2) * k ** -0.5, _rand(pairs, k, seed=3) * k ** -0.5
        proj.add("swiglu", interleave_rows(gate, up), n=pairs)
        outs.append(torch.full((m, pairs), float("nan"), device="cuda").bfloat16())
    proj.finish(torch.bfloat16, "cuda")
    proj(a, outs)
    ref = a.double() @ w.double().T
    # fp32 sums of k products of magnitude k^-1/2: k roundings of 2^-24 of a sum of about 1, in whatever order
    assert float((outs[0].double() - ref).abs().max()) < 8 * k ** 0.5 * 2 ** -24 * float(ref.abs().max())
    if pairs:
        g, u = a.double() @ gate.double().T, a.double() @ up.double().T
        want = torch.nn.functional.silu(g) * u
        # half a unit in the last of 8 bits, and what the fast exponential and division add
        assert float(((outs[1].double() - want).abs() - 2 ** -8 * want.abs()).max()) < 1e-4


@pytest.mark.parametrize("m", [2, 3, 8, 9, 64, 128])
@pytest.mark.parametrize("n,ks", [(1056, (136, 520)), (2048, (2048, 6144)), (4096, (4096,))])
def test_gated_update(m, n, ks):
    from flashrec_b200.lm_layers import gated_add

    x = torch.randn(m, n, device="cuda", generator=torch.Generator(device="cuda").manual_seed(5))
    parts = [(_rand(m, k, seed=k), _rand(n, k, seed=k + 1) * k ** -0.5, _rand(m, n, seed=k + 2)) for k in ks]
    want = x.double() + sum(g.double() * (a.double() @ w.double().T) for a, w, g in parts)
    p = gated_add(x, parts, few_rows=True)
    got = x.double() + (p.buf.double().sum(0) if p is not None else 0)
    assert float((got - want).abs().max()) < 8 * max(ks) ** 0.5 * 2 ** -24 * float(want.abs().max())

"""Few-row products around the lines where they change kernel, tile width and k-blocks per stage, against fp32."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _clean_status():
    yield
    from flashrec_b200 import device_status

    assert device_status() == (0, 0)


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


@pytest.mark.parametrize("m", [3, 4, 5, 7, 8])
@pytest.mark.parametrize("k", [2048, 2056, 12296])
@pytest.mark.parametrize("n,pairs", [(2052, 0), (3080, 0), (4100, 0), (5156, 544), (9476, 0), (32, 4128)])
def test_up_to_eight_rows_are_summed_in_fp32(m, k, n, pairs):
    """Long products of few rows, on either side of the line between the row kernel and the tensor cores."""
    from flashrec_b200 import device_status
    from flashrec_b200.lm_layers import MergedProjection, interleave_rows

    a, w = _rand(m, k, seed=m), _rand(n, k, seed=1) * k ** -0.5
    proj = MergedProjection(k)
    proj.add("store_f32", w)
    outs = [torch.full((m, n), float("nan"), device="cuda")]
    if pairs:
        gate, up = _rand(pairs, k, seed=2) * k ** -0.5, _rand(pairs, k, seed=3) * k ** -0.5
        proj.add("swiglu", interleave_rows(gate, up), n=pairs)
        outs.append(torch.full((m, pairs), float("nan"), device="cuda").bfloat16())
    proj.finish(torch.bfloat16, "cuda")
    proj(a, outs)
    ref = a.double() @ w.double().T
    # the result's own rounding is 2^-24 of an element at most, 0.6 of that in the norm; sums of k products in fp32 add about as
    # much, whatever k; accumulated in the tensor cores they would add 1e-9 of the norm per element of k, 2e-6 at the least here
    assert float((outs[0].double() - ref).norm() / ref.norm()) < 2 * 2 ** -24
    if pairs:
        g, u = a.double() @ gate.double().T, a.double() @ up.double().T
        want = torch.nn.functional.silu(g) * u
        assert float(((outs[1].double() - want).abs() - 2 ** -8 * want.abs()).max()) < 1e-4
    assert device_status() == (0, 0)


@pytest.mark.parametrize("m", [5, 8])
@pytest.mark.parametrize("n,ks", [(1056, (2056,)), (2048, (2048, 6144)), (4100, (12288,))])
def test_updates_of_up_to_eight_rows_are_summed_in_fp32(m, n, ks):
    from flashrec_b200 import device_status
    from flashrec_b200.lm_layers import gated_add, split_product

    parts = [(_rand(m, k, seed=k), _rand(n, k, seed=k + 1) * k ** -0.5, _rand(m, n + (-n) % 8, seed=k + 2)[:, :n]) for k in ks]
    x = torch.zeros(m, n, device="cuda")
    want = sum(g.double() * (a.double() @ w.double().T) for a, w, g in parts)
    p = gated_add(x, parts, few_rows=True)
    got = x.double() + (p.buf.double().sum(0) if p is not None else 0)
    assert float((got - want).norm() / want.norm()) < 2 * 2 ** -24
    p = split_product(*parts[0][:2])
    want = parts[0][0].double() @ parts[0][1].double().T
    assert p is None or float((p.buf.double().sum(0) - want).norm() / want.norm()) < 2 * 2 ** -24
    assert device_status() == (0, 0)


@pytest.mark.parametrize("m", [3, 8])
@pytest.mark.parametrize("n", [1056, 6148])
def test_few_rows_with_infinities_and_nan(m, n):
    from flashrec_b200.lm_layers import MergedProjection

    k = 4096
    a, w = _rand(m, k, seed=m), (_rand(n, k, seed=1).abs() + 0.5) * k ** -0.5
    a[0, 5], a[1, k - 1], a[2, 70], a[2, 4000] = float("inf"), float("-inf"), float("inf"), float("nan")
    proj = MergedProjection(k)
    proj.add("store_f32", w)
    proj.finish(torch.bfloat16, "cuda")
    out = torch.zeros((m, n), device="cuda")
    proj(a, [out])
    assert (out[0] == float("inf")).all() and (out[1] == float("-inf")).all() and out[2].isnan().all()
    assert out[3:].isfinite().all()


@pytest.mark.parametrize("m", [65, 129, 351])
@pytest.mark.parametrize("k", [504, 512, 1048])
def test_f32_tiles_of_128_rows(m, k):
    """Columns enough for a tile of 128 rows per SM, with pairs, rows left over, and K on either side of the line."""
    from flashrec_b200.lm_layers import MergedProjection, interleave_rows

    g = torch.Generator(device="cuda").manual_seed(k)
    r = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    plain, pairs = 8228, 912
    a, w, gate, up = r(m, k), r(plain, k) * k ** -0.5, r(pairs, k) * k ** -0.5, r(pairs, k) * k ** -0.5
    proj = MergedProjection(k)
    proj.add("store", w)
    proj.add("swiglu", interleave_rows(gate, up), n=pairs)
    proj.finish(torch.float32, "cuda")
    outs = [torch.full((m, plain), float("nan"), device="cuda"), torch.full((m, pairs), float("nan"), device="cuda")]
    proj(a, outs)
    for got, want in zip(outs, (a.double() @ w.double().T, torch.nn.functional.silu(a.double() @ gate.double().T) * (a.double() @ up.double().T))):
        # k roundings of 2^-24 of a sum of about 1 in random order, and a few more of the activation's
        assert float((got.double() - want).norm() / want.norm()) < (k ** 0.5 + 8) * 2 ** -24


@pytest.mark.parametrize("m", [9, 64, 65, 300, 1024, 1025])
@pytest.mark.parametrize("n,ks", [(1060, (520, 1544)), (2048, (2048, 6144)), (4096, (4096,)), (68, (1032,))])
def test_f32_updates_in_shares(m, n, ks):
    """K split over CTAs, up to 1024 rows, with rows, columns and steps of K left over."""
    from flashrec_b200 import lm_layers as L

    g = torch.Generator(device="cuda").manual_seed(m + n)
    r = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    x, parts = r(m, n), [(r(m, k), r(n, k) * k ** -0.5, r(m, n)) for k in ks]
    want = x.double() + sum(gt.double() * (a.double() @ w.double().T) for a, w, gt in parts)
    p = L.gated_add(x, parts, few_rows=True)
    assert (p is None) == (m > 1024 or -(-m // 64) * -(-n // 64) >= 888)
    got = x.double() + (p.buf.double().sum(0) if p is not None else 0)
    # k roundings of 2^-24 of sums of about 1 in random order, the gate's and the stream's
    assert float((got - want).norm() / want.norm()) < (max(ks) ** 0.5 + 4) * 2 ** -24


@pytest.mark.parametrize("m,n,k", [(385, 37888, 72), (700, 20480, 136), (1111, 10016, 520), (1923, 4128, 1096), (5000, 2080, 72)])
def test_pairs_of_ctas(m, n, k):
    """Tiles of 256 rows on two SMs, with rows, columns and K left over: a projection and an update in two parts."""
    from flashrec_b200.lm_layers import MergedProjection, gated_add

    a, w = _rand(m, k, seed=m), _rand(n, k, seed=1) * k ** -0.5
    proj = MergedProjection(k)
    proj.add("store_f32", w)
    proj.finish(torch.bfloat16, "cuda")
    out = torch.full((m, n), float("nan"), device="cuda")
    proj(a, [out])
    ref = a.double() @ w.double().T
    # as in test_projection: k roundings of 2^-24 of a sum of about 1, in whatever order
    bound = 8 * k ** 0.5 * 2 ** -24
    assert float((out.double() - ref).abs().max()) < bound * float(ref.abs().max())
    x, gate = torch.randn(m, n, device="cuda", generator=torch.Generator(device="cuda").manual_seed(5)), _rand(m, n, seed=2)
    want = x.double() + gate.double() * ref + ref
    assert gated_add(x, [(a, w, gate), (a, w, None)], split=False) is None
    assert float((x.double() - want).abs().max()) < 2 * bound * float(want.abs().max())


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("m,n,ks", [(1, 2056, (264, 520)), (2, 4096, (6144,)), (4, 520, (2048, 72)), (64, 2048, (2048, 6144)),
                                    (130, 776, (1096,)), (700, 20480, (136,))])
def test_weights_read_ahead_of_the_launch_before_keep_the_bits(dtype, m, n, ks):
    """The activations come from a launch that ends while the product begins."""
    from flashrec_b200.lm_layers import gated_add, rms_norm

    h = [_rand(m, k, seed=k).float() for k in ks]
    ws = [(_rand(n, k, seed=i) * k ** -0.5).to(dtype) for i, k in enumerate(ks)]
    x0, got = torch.randn(m, n, device="cuda", generator=torch.Generator(device="cuda").manual_seed(5)), []
    for laid_out in (True, False):
        x = x0.clone()
        for split in (False, True):
            acts = [torch.empty(m, k, dtype=dtype, device="cuda") for k in ks]
            for a, v, k in zip(acts, h, ks):
                rms_norm(v, torch.ones(k, device="cuda"), 0.0, 1e-6, a)
            p = gated_add(x, [(a, w, None) for a, w in zip(acts, ws)], few_rows=True, split=split, laid_out=laid_out)
            if p is not None:
                got.append(p.buf)
        got.append(x)
    for a, b in zip(got[: len(got) // 2], got[len(got) // 2:]):
        assert torch.equal(a, b)


@pytest.mark.parametrize("dtype,m", [(torch.bfloat16, 1), (torch.bfloat16, 2), (torch.bfloat16, 64), (torch.bfloat16, 600), (torch.float32, 1)])
def test_projection_of_a_weight_that_the_launch_ahead_writes(dtype, m):
    """The weight comes from a product that lets its dependents start at its own beginning: a projection whose caller does not
    say that it lies there already sees all of it."""
    from flashrec_b200.lm_layers import MergedProjection

    n, k, depth = 1064, 512, 4096
    proj = MergedProjection(k)
    proj.add("store_f32", torch.zeros(n, k))
    proj.finish(dtype, "cuda")
    writer = MergedProjection(depth)
    writer.add("store", _rand(k, depth, seed=1) * depth ** -0.5)
    writer.finish(dtype, "cuda")
    a = _rand(m, k, seed=2).to(dtype)
    inputs = [_rand(n, depth, seed=10 + i).to(dtype) for i in range(16)]
    torch.cuda.synchronize()

    def step(x, wait=False):
        writer(x, [proj.weight[:n]])
        if wait:
            torch.cuda.synchronize()
        out = torch.empty(m, n, device="cuda")
        proj(a, [out])
        return out

    want = [step(x, wait=True) for x in inputs]
    assert not torch.equal(want[0], want[1])
    for _ in range(3):
        torch.cuda._sleep(20_000_000)  # the launches queue up and meet the GPU without gaps
        for got, ref in zip([step(x) for x in inputs], want):
            assert torch.equal(got, ref)

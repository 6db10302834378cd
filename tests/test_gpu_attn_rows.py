"""Row attention of bf16 heads up to 128 (one launch) against the general kernels, which the same call takes in float32:
every mixture over rows of unequal length, at the edges of its key blocks, warps, shares and clusters."""

import pytest
import torch

pytestmark = pytest.mark.gpu

PAGE = 64


def _run(kind, dtype, heads, kv, dim, vdim, lens, window, keep, seed, edit=None, slopes=None):
    """One query per request, at the last of its ``lens`` tokens; [rows, heads * vdim] as float."""
    from flashrec_b200.core import ForwardBatch
    from flashrec_b200.kvcache import CacheSpec
    from flashrec_b200.lm_layers import MixAttention, alibi_slopes

    maps = 2 if kind == "diff" else 1
    g = torch.Generator().manual_seed(seed)
    rnd = lambda *s: torch.randn(*s, generator=g).bfloat16()  # noqa: E731
    n, pages = len(lens), [(m + PAGE - 1) // PAGE for m in lens]
    perm, table, at = torch.randperm(sum(pages), generator=g), torch.zeros((n + 1, max(pages) * PAGE), dtype=torch.int32), 0
    for r, p in enumerate(pages):
        table[r + 1, :p * PAGE] = (perm[at:at + p, None] * PAGE + torch.arange(PAGE)).reshape(-1).to(torch.int32)
        at += p
    slots = sum(pages) * PAGE
    q, k, v = rnd(n, heads * maps * dim), rnd(slots, kv * maps * dim), rnd(slots, kv * vdim)
    if edit is not None:
        edit(q, k, table[1:].long())
    coef, gate = 0.5 * torch.randn(heads, heads, generator=g), torch.randn(n, heads, generator=g)
    if kind == "talk":
        slopes = torch.tensor(alibi_slopes(heads))
    spec = CacheSpec(0, 0, mask="chunk" if kind == "talk" else "window", size=window, keep_first=keep)
    attn = MixAttention(kind, heads, kv, dim, vdim, dim ** -0.5, spec, eps=1e-5, lam=0.4, out_scale=0.8,
                        coef=coef if kind == "talk" else None, slopes=slopes)
    attn.bind("cuda")
    pos = torch.tensor([m - 1 for m in lens])
    b = ForwardBatch(input_ids=None, req_pool_indices=torch.arange(1, n + 1).cuda(), seq_lens=None, positions=pos.cuda(),
                     tok_req=torch.arange(n, dtype=torch.int32).cuda(), n_row_tokens=n, max_pos=max(lens) - 1)
    counters = torch.zeros(4096, dtype=torch.int32, device="cuda")
    y = attn.forward(*(x.to(dtype).cuda() for x in (q, k, v)), table.cuda(), b, counters,
                     head_gate=gate.cuda() if kind == "plain" else None)
    assert not counters.any()
    return y.float().cpu()


@pytest.mark.parametrize("kind", ["diff", "talk", "plain"])
@pytest.mark.parametrize("heads,kv,dim,vdim", [(16, 8, 128, 128), (4, 4, 64, 128), (8, 2, 64, 64), (8, 1, 128, 48), (4, 2, 64, 48), (6, 2, 80, 128), (5, 1, 16, 16)])
@pytest.mark.parametrize("lens,window,keep", [
    ((1,), 4096, 0), ((1100,), 4096, 0), ((3000,), 1024, 4), ((31, 32, 33, 1, 127, 128, 129, 257), 200, 3),
    (tuple(range(5, 400, 9)), 300, 1)])
def test_rows_match_the_general_kernels(kind, heads, kv, dim, vdim, lens, window, keep):
    if kind != "diff" and keep:
        keep = 0
    got, ref = (_run(kind, d, heads, kv, dim, vdim, lens, window, keep, 3) for d in (torch.bfloat16, torch.float32))
    # both compute in fp32 from the same values; rounding to the 8 significant bits of bf16 moves each element by at most half
    # a unit in the last place, 2^-8 of it, and sums in another order move the norm by a few 1e-6
    err = (got - ref).norm(dim=1) / ref.norm(dim=1)
    assert err.max() < 2 ** -8 + 1e-4, (int(err.argmax()), float(err.max()))


@pytest.mark.parametrize("kind", ["diff", "talk", "plain"])
@pytest.mark.parametrize("value", [float("-inf"), float("nan")])
@pytest.mark.parametrize("n,at", [(33, [32]), (97, [96]), (100, list(range(32))), (300, [40, 299]), (1100, [1099]), (1100, list(range(160, 192)))])
def test_keys_that_are_not_finite(kind, value, n, at):
    """Keys whose score is -inf weigh nothing, wherever the first of them stands in the walk; a NaN reaches the output."""
    def edit(q, k, slots):
        q[:, ::64] = q[:, ::64].abs() + 0.5
        for p in at:
            k[slots[0][p], ::64] = value

    got, ref = (_run(kind, d, 4, 2, 64, 64, (n, 20), 4096, 0, 5, edit) for d in (torch.bfloat16, torch.float32))
    bad = torch.isnan(ref[0]).all() if value != value else torch.isfinite(ref[0]).all()
    assert bad and torch.equal(torch.isnan(got), torch.isnan(ref))
    got, ref = got.nan_to_num(0.0), ref.nan_to_num(0.0)
    assert ((got - ref).norm(dim=1) <= (2 ** -8 + 1e-4) * ref.norm(dim=1)).all()


@pytest.mark.parametrize("kind", ["diff", "talk", "plain"])
def test_sums_are_as_accurate_as_the_general_kernels(kind):
    """How often an output is not the bf16 nearest to the 64-bit result: that share grows with the error before rounding. 10^6
    outputs per kernel and 2 to 3 in 10^4 of them: the ratio of two such counts is known to 9 %."""
    from flashrec_b200.core import ForwardBatch
    from flashrec_b200.kvcache import CacheSpec
    from flashrec_b200.lm_layers import MixAttention

    n, m, heads, kv, vdim, dim = 32, 832, 16, 8, 128, 64 if kind == "diff" else 128
    maps, scale = 2 if kind == "diff" else 1, dim ** -0.5
    coef = 0.5 * torch.randn(heads, heads, generator=torch.Generator().manual_seed(0))
    attn = MixAttention(kind, heads, kv, dim, vdim, scale, CacheSpec(0, 0, size=4096), eps=1e-5, lam=0.5, out_scale=1.0,
                        coef=coef if kind == "talk" else None)
    attn.bind("cuda")
    table = torch.cat([torch.zeros(1, m), torch.arange(n * m).view(n, m)]).to(torch.int32).cuda()
    b = ForwardBatch(input_ids=None, req_pool_indices=torch.arange(1, n + 1).cuda(), seq_lens=None, positions=torch.full((n,), m - 1).cuda(),
                     tok_req=torch.arange(n, dtype=torch.int32).cuda(), n_row_tokens=n, max_pos=m - 1)
    counters, off = torch.zeros(4096, dtype=torch.int32, device="cuda"), {torch.bfloat16: 0, torch.float32: 0}
    for seed in range(16):
        g = torch.Generator(device="cuda").manual_seed(seed)
        q, k, v = (torch.randn(*s, generator=g, device="cuda").bfloat16() for s in ((n, heads * maps * dim), (n * m, kv * maps * dim), (n * m, kv * vdim)))
        qd = q.double().view(n, kv, heads // kv, maps, dim)
        p = torch.softmax(scale * torch.einsum("ngrad,nkgad->ngrak", qd, k.double().view(n, m, kv, maps, dim)), -1)
        p = p[..., 0, :] - 0.5 * p[..., 1, :] if kind == "diff" else p[..., 0, :]
        if kind == "talk":
            p = torch.einsum("os,nsk->nok", coef.double().cuda(), p.reshape(n, heads, m)).view_as(p)
        want = torch.einsum("ngrk,nkgd->ngrd", p, v.double().view(n, m, kv, vdim))
        if kind == "diff":
            want = want * (want.pow(2).mean(-1, keepdim=True) + 1e-5).rsqrt()
        for dtype in off:
            got = attn.forward(*(x.to(dtype) for x in (q, k, v)), table, b, counters).bfloat16()
            off[dtype] += int((got != want.view(n, -1).bfloat16()).sum())
    assert off[torch.float32] > 100 and off[torch.bfloat16] < 1.18 * off[torch.float32], off


@pytest.mark.parametrize("kind,maps", [("diff", 2), ("plain", 1)])
@pytest.mark.parametrize("heads,kv,lens", [(4, 4, (1, 33, 700)), (8, 2, (129, 1500)), (6, 2, tuple(range(5, 300, 9)))])
def test_slopes_of_every_map(kind, maps, heads, kv, lens):
    slopes = 0.3 * torch.rand(heads * maps, generator=torch.Generator().manual_seed(1))
    got, ref = (_run(kind, d, heads, kv, 64, 64, lens, 4096, 0, 7, slopes=slopes) for d in (torch.bfloat16, torch.float32))
    assert ((got - ref).norm(dim=1) < (2 ** -8 + 1e-4) * ref.norm(dim=1)).all()


@pytest.mark.parametrize("kind", ["diff", "talk", "plain"])
@pytest.mark.parametrize("heads,kv", [(4, 2), (8, 1), (6, 2)])
@pytest.mark.parametrize("scratch", [0, 300_000])
def test_rows_of_a_batch_that_is_cut(kind, heads, kv, scratch, monkeypatch):
    """Scratch for a row or a few at a time: the launches begin behind the batch's first row."""
    from flashrec_b200 import lm_layers

    lens = tuple(range(5, 400, 9))
    ref = _run(kind, torch.float32, heads, kv, 64, 64, lens, 300, 0, 9)
    monkeypatch.setattr(lm_layers, "_SCORE_SCRATCH_BYTES", scratch)
    begins, call = [], lm_layers.call
    monkeypatch.setattr(lm_layers, "call", lambda name, *a: begins.append((name, a[1])) or call(name, *a))
    got = _run(kind, torch.bfloat16, heads, kv, 64, 64, lens, 300, 0, 9)
    assert [n for n, _ in begins].count("fr_mix_attn_rows") > 1 and max(r for _, r in begins) > 20
    assert ((got - ref).norm(dim=1) < (2 ** -8 + 1e-4) * ref.norm(dim=1)).all()


@pytest.mark.parametrize("kind", ["diff", "talk", "plain"])
@pytest.mark.parametrize("heads,kv,dim,vdim", [(16, 8, 128, 128), (8, 2, 64, 64), (5, 1, 16, 16)])
@pytest.mark.parametrize("lens", [(1,), (1100,), (15, 16, 17, 18, 31, 33, 129, 257)])
def test_reads_before_the_launch_ahead_has_ended(kind, heads, kv, dim, vdim, lens, monkeypatch):
    """The early entry, with everything written long before, gives the same bits."""
    from flashrec_b200 import lm_layers

    ref = _run(kind, torch.bfloat16, heads, kv, dim, vdim, lens, 200, 0, 11)
    call = lm_layers.call

    def early(name, *a):
        torch.cuda.synchronize()
        call(name + "_early" if name == "fr_mix_attn_rows" else name, *a)

    monkeypatch.setattr(lm_layers, "call", early)
    assert torch.equal(_run(kind, torch.bfloat16, heads, kv, dim, vdim, lens, 200, 0, 11), ref)


def _decode(kind, heads, kv, dim, vdim, lens):
    """A bound attention and a batch of one query per request, at the last of its ``lens`` tokens; pages lie one after the other."""
    from flashrec_b200.core import ForwardBatch
    from flashrec_b200.kvcache import CacheSpec
    from flashrec_b200.lm_layers import MixAttention

    n, pages = len(lens), [(m + PAGE - 1) // PAGE for m in lens]
    table, at = torch.zeros((n + 1, max(pages) * PAGE), dtype=torch.int32), 0
    for r, p in enumerate(pages):
        table[r + 1, :p * PAGE] = torch.arange(at, at + p * PAGE)
        at += p * PAGE
    attn = MixAttention(kind, heads, kv, dim, vdim, dim ** -0.5, CacheSpec(0, 0, size=4096), eps=1e-5, lam=0.4, out_scale=0.8,
                        coef=torch.zeros(heads, heads) if kind == "talk" else None)
    attn.bind("cuda")
    pos = torch.tensor([m - 1 for m in lens])
    b = ForwardBatch(input_ids=None, req_pool_indices=torch.arange(1, n + 1).cuda(), seq_lens=None, positions=pos.cuda(),
                     out_cache_loc=table[torch.arange(1, n + 1), pos].long().cuda(),
                     tok_req=torch.arange(n, dtype=torch.int32).cuda(), n_row_tokens=n, max_pos=max(lens) - 1)
    return attn, table.cuda(), b, at


def _behind_each_other(step, inputs):
    """``step`` over the inputs, queued behind a sleep, so that the GPU meets the launches without gaps."""
    torch.cuda._sleep(20_000_000)
    return [step(x) for x in inputs]


@pytest.mark.parametrize("heads,kv,lens", [(8, 4, (300,)), (8, 8, (700, 33)), (16, 8, tuple(range(20, 420, 10)))])
def test_coefficients_of_the_launch_ahead(heads, kv, lens):
    """The mixing matrix comes from a product that lets its dependents start at its own beginning: the plain entry sees all of it."""
    from flashrec_b200.lm_layers import MergedProjection

    n, dim, depth = len(lens), 64, 8192
    attn, table, b, slots = _decode("talk", heads, kv, dim, dim, lens)
    g = torch.Generator(device="cuda").manual_seed(heads)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda").bfloat16()  # noqa: E731
    q, k, v = rnd(n, heads * dim), rnd(slots, kv * dim), rnd(slots, kv * dim)
    proj = MergedProjection(depth)
    proj.add("store_f32", rnd(heads, depth) * depth ** -0.5)
    proj.finish(torch.bfloat16, "cuda")
    torch.cuda.synchronize()
    counters, inputs = torch.zeros(4096, dtype=torch.int32, device="cuda"), [rnd(heads, depth) for _ in range(24)]

    def step(x, wait=False):
        proj(x, [attn.coef])
        if wait:
            torch.cuda.synchronize()
        return attn.forward(q, k, v, table, b, counters)

    want = [step(x, wait=True) for x in inputs]
    assert not torch.equal(want[0], want[1])
    for _ in range(3):
        for got, ref in zip(_behind_each_other(step, inputs), want):
            assert torch.equal(got, ref)


@pytest.mark.parametrize("kind", ["diff", "talk", "plain"])
@pytest.mark.parametrize("lens", [(1100,), (1,), tuple(range(40, 440, 10))])
def test_early_reads_behind_a_launch_that_writes(kind, lens):
    """Queries, the rows' own keys and values and the heads' gates come, over the same buffers again and again, from a product that
    lets its dependents start at its own beginning: the early entry's bits are those of the plain one behind a wait."""
    from flashrec_b200.lm_layers import MergedProjection

    n, heads, kv, dim, vdim, depth = len(lens), 8, 4, 64, 128, 4096
    maps = 2 if kind == "diff" else 1
    attn, table, b, slots = _decode(kind, heads, kv, dim, vdim, lens)
    g = torch.Generator(device="cuda").manual_seed(n)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda").bfloat16()  # noqa: E731
    if kind == "talk":
        attn.coef.copy_(0.5 * rnd(heads, heads).float())
    q, k, v, gate = rnd(n, heads * maps * dim), rnd(slots, kv * maps * dim), rnd(slots, kv * vdim), torch.zeros(n, heads, device="cuda")
    proj = MergedProjection(depth)
    for cols, store in ((q.shape[1], "store"), (k.shape[1], "store"), (v.shape[1], "store"), (heads, "store_f32")):
        proj.add(store, rnd(cols, depth) * 4 * depth ** -0.5)
    proj.finish(torch.bfloat16, "cuda")
    torch.cuda.synchronize()
    counters, inputs = torch.zeros(4096, dtype=torch.int32, device="cuda"), [rnd(n, depth) for _ in range(24)]

    def step(x, wait=False):
        proj(x, [q, k, v, gate], [None, b.out_cache_loc, b.out_cache_loc, None], laid_out=True)
        if wait:
            torch.cuda.synchronize()
        return attn.forward(q, k, v, table, b, counters, head_gate=gate if kind == "plain" else None, early=not wait)

    want = [step(x, wait=True) for x in inputs]
    assert not torch.equal(want[0], want[1])
    for _ in range(3):
        for got, ref in zip(_behind_each_other(step, inputs), want):
            assert torch.equal(got, ref)

"""Host side of the step function: slots of many positions at once as one by one, tokens in every form."""

import random

import numpy as np
import pytest
import torch

from flashrec_b200.engine import _token_array
from flashrec_b200.kvcache import PAGE, CacheSpec, SequenceManager


def test_slots_of_many_positions_are_those_of_one_after_the_other():
    r = random.Random(0)
    one, many = (SequenceManager([CacheSpec(8, 8)], 60, 4, 2000, "cpu") for _ in range(2))
    for m in (one, many):
        for q in range(3):
            m.open(q)
    for _ in range(200):
        q, n = r.randrange(3), r.choice([0, 1, 2, PAGE - 1, PAGE, PAGE + 1, 130])
        try:
            slots = one.extend(q, n)
        except RuntimeError:
            with pytest.raises(RuntimeError):
                many.extend_array(q, n)
            for m in (one, many):
                m.close(q)
                m.open(q)
            continue
        assert slots == many.extend_array(q, n).tolist()
        assert one.length(q) == many.length(q) and one._free_pages == many._free_pages


@pytest.mark.parametrize("tokens", [[1, 99], (0, 4), range(5), np.array([1, 2], np.uint8), np.array([7], np.int32), torch.tensor([1, 2]),
                                    [np.int32(4), 7], [torch.tensor(3), 4], [1.0, 2], [True, 5]])
def test_tokens_in_every_form(tokens):
    a = _token_array(tokens, 100)
    assert a.dtype == np.int64 and a.tolist() == [int(t) for t in tokens]


@pytest.mark.parametrize("tokens", [[1, -1], [5, 100], (2 ** 70, 1), np.array([3, 200]), torch.tensor([1, 100]), np.array([2 ** 63], np.uint64)])
def test_tokens_outside_the_vocabulary(tokens):
    with pytest.raises(ValueError):
        _token_array(tokens, 100)


@pytest.mark.parametrize("tokens", [[torch.tensor(3.0, requires_grad=True), 4], (torch.tensor([3]), torch.tensor([4]))])
def test_tokens_that_are_no_arrays(tokens):
    a = _token_array(tokens, 100)  # NumPy takes neither list as a column of integers, the first not at all
    assert a.dtype == np.int64 and a.tolist() == [3, 4]


def test_single_tokens_in_every_container(monkeypatch):
    from types import SimpleNamespace

    from flashrec_b200.engine import LMEngine, StepEntry

    model = SimpleNamespace(device="cpu", vocab=100, cache_specs=[CacheSpec(8, 8)], new_caches=lambda *_: None)
    eng = LMEngine(model, 256, 4)
    got = []
    monkeypatch.setattr(LMEngine, "_decode", lambda self, toks, *_: got.append(list(toks)) or torch.zeros(0, 100))
    eng.step([StepEntry(i, t) for i, t in enumerate(([7], {8}, {9: "x"}.keys(), torch.tensor([10])))])
    assert got == [[7, 8, 9, 10]]


def _host_engine(max_tokens, reqs):
    from types import SimpleNamespace

    from flashrec_b200.engine import LMEngine

    model = SimpleNamespace(device="cpu", vocab=1000, cache_specs=[CacheSpec(8, 8)], new_caches=lambda *_: None,
                            forward=lambda *_, **__: (None, None))
    return LMEngine(model, max_tokens, reqs, use_graphs=False)


@pytest.mark.parametrize("lens", [[1] * 20 + [300], [200, 1, 9, 8, 130, 2, 127, 128, 1], [3, 9, 64], [1, 1], [128]])
def test_columns_of_mixed_entries(lens, monkeypatch):
    from flashrec_b200.engine import ARRAY_TOKENS, LMEngine, StepEntry
    from flashrec_b200.lm_layers import ROW_PORTION

    eng, got, arrays = _host_engine(4096, len(lens)), [], []
    take = eng.seqs.extend_array
    monkeypatch.setattr(eng.seqs, "extend_array", lambda req, n: arrays.append(n) or take(req, n))
    seen = lambda: {i: (s.row, dict(s.pages)) for i, s in eng.seqs.live.items()}  # pages behind a window leave after the step
    monkeypatch.setattr(LMEngine, "_stage", lambda self, *a: got.append((a, seen())) or (None, None))
    for step in range(2):
        entries = [StepEntry(i, [(31 * i + 7 * t + step) % 1000 for t in range(n)]) for i, n in enumerate(lens)]
        first = [eng.seqs.length(e.req) for e in entries]
        eng.step(entries)
        (toks, pos, loc, rows, req_rows, want, tok_req, qo, pre, ext, tiles, n_row, one), held = got.pop()
        order = sorted(range(len(lens)), key=lambda i: lens[i] > ROW_PORTION)
        assert list(toks) == [t for i in order for t in entries[i].tokens]
        assert list(pos) == [first[i] + t for i in order for t in range(lens[i])]
        assert list(tok_req) == [b for b, i in enumerate(order) for _ in range(lens[i])]
        assert list(rows) == [held[i][0] for i in order for _ in range(lens[i])]
        assert list(loc) == [held[i][1][p // PAGE] * PAGE + p % PAGE for i in order for p in range(first[i], first[i] + lens[i])]
    assert sorted(arrays) == sorted(2 * [n for n in lens if n >= ARRAY_TOKENS])  # what an array costs, only long entries repay

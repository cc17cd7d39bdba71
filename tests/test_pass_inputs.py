"""Inputs of a pass: numbers from the host's lists, and a session's steps against passes described by set_rows()."""
import collections

import numpy as np
import pytest
import torch

from ds41rt_b200.models.base import row_values


@pytest.mark.parametrize("values", [[], [7], list(range(5, 69)), range(3, 67), range(10, 0, -3), (1, 2, 3), [True, False],
                                    [2 ** 31 - 1, -2 ** 31], [1.9, -1.9], torch.arange(9), list(torch.arange(4)),
                                    bytes(range(97, 105)), bytearray(4), range(7, 7), range(2 ** 31 - 3, 2 ** 31 - 1),
                                    torch.tensor([3, 4], dtype=torch.int32), np.arange(5)])
def test_row_values(values):
    want = torch.tensor(list(values) + [-1] * (64 - len(values)), dtype=torch.int32)
    assert torch.equal(row_values(values, 64, -1), want)


def test_row_values_refused():
    with pytest.raises(RuntimeError):
        row_values([2 ** 31], 4, 0)
    with pytest.raises(RuntimeError):
        row_values([1, 2, 3], 2, 0)


@pytest.mark.parametrize("values", [torch.tensor([2 ** 31]), range(2 ** 31 - 1, 2 ** 31 + 1), range(-2 ** 31 - 1, -2 ** 31),
                                    [float("nan")], (0, -2 ** 31 - 1)])
def test_numbers_that_do_not_fit(values):
    with pytest.raises(RuntimeError):
        row_values(values, 2, 0)


def _host_rows(kind, rows):
    """An engine that has nothing but the inputs of a pass, on the CPU."""
    from ds41rt_b200.models.ds41 import DS41Engine
    from ds41rt_b200.models.stack import StackEngine
    e = object.__new__(StackEngine if kind == "stack" else DS41Engine)
    e.max_rows, e.long_rows, e.f32, e.moe_rows, e.max_keys, e.idx_q = rows, 4, 0, 4, 64, None
    e.in_tokens, e.row_pos, e.row_slot, e.row_lo, e.row_hi = torch.zeros(5, rows, dtype=torch.int32).unbind()
    return e


@pytest.mark.parametrize("kind", ["stack", "flash"])
@pytest.mark.parametrize("rows", [8, 600])
def test_set_rows_takes_what_yields_numbers(kind, rows):
    e = _host_rows(kind, rows)
    e.set_rows(b"abc", collections.deque([4, 5, 9]), iter([0, 0, 1]))
    pad = [0] * (rows - 3)
    assert e.in_tokens.tolist() == [97, 98, 99] + pad and e.row_pos.tolist() == [4, 5, 9] + pad
    assert e.row_slot.tolist() == [0, 0, 1] + [-1] * (rows - 3)


def test_requests_of_a_pass(monkeypatch):
    """The loop over few rows and the array operations over many, against the rule stated plainly."""
    from ds41rt_b200.models import stack

    def plain(pos, slot):
        for s in set(slot) - {-1}:
            at = [i for i, x in enumerate(slot) if x == s]
            if at != list(range(at[0], at[-1] + 1)) or [pos[i] for i in at] != list(range(pos[at[0]], pos[at[0]] + len(at))):
                return None
        return len(set(slot) - {-1})

    g, kinds = torch.Generator().manual_seed(5), set()
    for _ in range(600):
        n = int(torch.randint(0, 9, (1,), generator=g))
        slot = torch.randint(-1, 3, (n,), generator=g).sort(descending=bool(torch.randint(0, 2, (1,), generator=g))).values
        if torch.rand(1, generator=g) < 0.2:
            slot = slot[torch.randperm(n, generator=g)]
        pos = torch.arange(n) + 7
        if torch.rand(1, generator=g) < 0.3 and n:
            pos[int(torch.randint(0, n, (1,), generator=g))] += 1
        want = plain(pos.tolist(), slot.tolist())
        kinds.add(want)
        for line in (1000, -1):
            monkeypatch.setattr(stack, "LOOP_ROWS", line)
            rows = (pos.int().numpy(), slot.int().numpy())
            if want is None:
                with pytest.raises(AssertionError):
                    stack.row_requests(*rows)
            else:
                assert stack.row_requests(*rows) == want
    assert kinds == {None, 0, 1, 2, 3}


def _stack(rows):
    from ds41rt_b200.models import registry
    fam, cfg = registry.preset("genesun-tiny")
    dev = torch.device("cuda", 0)
    return lambda: fam.engine(cfg, fam.random_weights(cfg, dev), max_rows=rows, slots=4, max_ctx=128)


@pytest.mark.gpu
def test_refused_rows():
    e = _stack(8)()
    for pos, slot in (([0, 2], [0, 0]), ([0, 1, 1], [0, 1, 0]), ([0, 1, 1], [0, -1, 0])):
        with pytest.raises(AssertionError):
            e.set_rows([1] * len(pos), pos, slot)
    e.set_rows([1] * 4, [0, 9, 3, 4], [1, -1, 0, 0])
    assert e.row_slot.tolist() == [1, -1, 0, 0, -1, -1, -1, -1] and e.row_pos.tolist() == [0, 9, 3, 4, 0, 0, 0, 0]


@pytest.mark.gpu
@pytest.mark.parametrize("graphs", [False, True])
@pytest.mark.parametrize("n", [1, 3, 4])
def test_step_is_the_pass(graphs, n):
    from ds41rt_b200.runtime.session import DecodeSession
    got = []
    for by_step in (False, True):
        torch.manual_seed(1)
        e = _stack(4)()
        session = DecodeSession(e, use_graphs=graphs)
        for s in range(n):
            assert e.cache.ensure(s, 16)
        tokens, out = list(range(11, 11 + n)), []
        for pos in range(4):
            rows = (tokens, [pos] * n, list(range(n)))
            if by_step:
                tokens = session.step(*rows)
            else:
                e.set_rows(*rows)
                e.forward_rows(n)
                tokens = e.chosen[:n].tolist()
            out.append((tokens, e.logits_rows(n).clone()))
        with pytest.raises(ValueError):
            session.step([], [], [])
        with pytest.raises(ValueError):
            session.step([1] * 5, [9] * 5, list(range(5)))
        got.append(out)
    for (a, x), (b, y) in zip(*got):
        assert a == b and torch.equal(x, y)


def test_rehearsal_has_no_slots():
    """The eager pass before a graph's capture may see rows that an earlier pass left: none of them may own a slot."""
    from ds41rt_b200.models.base import RowsEngine
    e = RowsEngine()
    e.in_tokens, e.row_pos, e.row_slot = torch.tensor([3, 4]), torch.tensor([7, 8]), torch.tensor([0, 1])
    with e.rehearsal():
        assert e.row_slot.tolist() == [-1, -1]
        e.in_tokens += 1
        e.row_pos += 1
    assert (e.in_tokens.tolist(), e.row_pos.tolist(), e.row_slot.tolist()) == ([3, 4], [7, 8], [0, 1])


@pytest.mark.gpu
@pytest.mark.parametrize("experts,kv", [("bf16", "bf16"), ("mxfp8", "fp8")])
@pytest.mark.parametrize("length", [9, 17])
def test_first_steps_leave_other_rows_alone(length, experts, kv):
    """A session's first step of a row count makes its graph: the rows of earlier passes, in the step's places, are neither
    stepped again nor written anywhere.  One request alone beyond its ring, then both for the first time."""
    from ds41rt_b200.config import ModelConfig
    from ds41rt_b200.models.ds41 import DS41Engine, EngineWeights
    from ds41rt_b200.runtime.session import DecodeSession
    cfg, dev = ModelConfig.tiny(), torch.device("cuda", 0)
    w = EngineWeights.random(cfg, 0, 1, dev, seed=3, expert_dtype=experts)
    prompts = torch.randint(3, cfg.vocab, (2, 2 * length), generator=torch.Generator().manual_seed(length))
    alone, both = cfg.window + 24, 5
    got = []
    for graphs in (True, False):
        e = DS41Engine(cfg, w, max_rows=24, slots=2, max_ctx=256, kv_dtype=kv)
        session = DecodeSession(e, use_graphs=graphs)
        last, out = [], []
        for slot in (0, 1):
            assert e.cache.ensure(slot, 200)
            last.append(e.prefill(slot, prompts[slot, :length].tolist()))
        at = [length, length]
        for step in range(alone + both):
            slots = [1] if step < alone else [0, 1]
            tokens = session.step([last[s] for s in slots], [at[s] for s in slots], slots)
            for s, t in zip(slots, tokens):
                last[s] = t
                at[s] += 1
            out.append(e.logits_rows(len(slots)).clone())
        e.check_status()
        got.append((out, e.cache.win, [e.cache.comp[s] for s in e.cache.comp], [e.cache.idx[s] for s in e.cache.idx],
                    [e.cache.pending[s] for s in e.cache.pending]))
    (out, *caches), (want, *there) = got
    for i, (a, b) in enumerate(zip(out, want)):
        assert torch.equal(a, b), f"step {i}"
    flat = lambda c: [c[0], *c[1], *c[2], *c[3]]
    for a, b in zip(flat(caches), flat(there)):
        assert torch.equal(a.view(torch.uint8), b.view(torch.uint8))


@pytest.mark.gpu
@pytest.mark.parametrize("model", ["genesun-tiny", "belasun-tiny", "flash"])
def test_device_loop_without_graphs(model):
    """Steps whose tokens and positions are fed on the device, launched one by one far ahead of the GPU, against captured ones."""
    from ds41rt_b200.runtime.session import DecodeSession
    dev, n, steps = torch.device("cuda", 0), 3, 20
    if model == "flash":
        from ds41rt_b200.config import ModelConfig
        from ds41rt_b200.models.ds41 import DS41Engine, EngineWeights
        cfg = ModelConfig.tiny()
        w = EngineWeights.random(cfg, 0, 1, dev, seed=3)
        make = lambda: DS41Engine(cfg, w, max_rows=24, slots=n, max_ctx=256)
    else:
        from ds41rt_b200.models import registry
        fam, cfg = registry.preset(model)
        torch.manual_seed(2)
        w = fam.random_weights(cfg, dev)
        make = lambda: fam.engine(cfg, w, max_rows=24, slots=n, max_ctx=256)
    prompts = torch.randint(3, cfg.vocab, (n, 60), generator=torch.Generator().manual_seed(4))
    got = []
    for graphs in (True, False):
        e = make()
        session, last = DecodeSession(e, use_graphs=graphs), []
        for s in range(n):
            assert e.cache.ensure(s, 120)
            last.append(e.prefill(s, prompts[s, :40 + 10 * s].tolist(), chunk=20))
        e.set_rows(last, [40 + 10 * s for s in range(n)], list(range(n)))
        torch.cuda.synchronize()
        torch.cuda._sleep(20_000_000)                  # the launches are queued before the first one runs
        session.run_device_loop(n, steps)
        torch.cuda.synchronize()
        e.check_status()
        assert e.row_pos[:n].tolist() == [40 + 10 * s + steps for s in range(n)]
        got.append((e.in_tokens[:n].clone(), e.logits_rows(n).clone()))
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])

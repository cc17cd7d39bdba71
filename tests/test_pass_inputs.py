"""Inputs of a pass: numbers from the host's lists, and a session's steps against passes described by set_rows()."""
import pytest
import torch

from ds41rt_b200.models.base import row_values


@pytest.mark.parametrize("values", [[], [7], list(range(5, 69)), range(3, 67), range(10, 0, -3), (1, 2, 3), [True, False],
                                    [2 ** 31 - 1, -2 ** 31], [1.9, -1.9], torch.arange(9), list(torch.arange(4))])
def test_row_values(values):
    want = torch.tensor(list(values) + [-1] * (64 - len(values)), dtype=torch.int32)
    assert torch.equal(row_values(values, 64, -1), want)


def test_row_values_refused():
    with pytest.raises(RuntimeError):
        row_values([2 ** 31], 4, 0)
    with pytest.raises(RuntimeError):
        row_values([1, 2, 3], 2, 0)


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

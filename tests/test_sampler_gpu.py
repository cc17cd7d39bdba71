"""GPU sampler against the host oracle: every filter combination, masks, ties, error statuses."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _oracle(logits, mask, p):
    from ds41rt_b200.runtime import core
    u = core.sample_uniform(p.seed, p.position)
    try:
        return core.sample_token(logits, mask, p.temperature, p.top_k, p.top_p, p.min_p, u), 0
    except core.SamplingError as e:
        return -1, str(e)


@pytest.mark.parametrize("vocab", [1000, 4096, 129280])
def test_sampler_matches_host_oracle(vocab):
    from ds41rt_b200.ops.sampling import RowParams, pack_params, sample_rows
    rng = np.random.default_rng(vocab)
    combos = [dict(temperature=0.0), dict(temperature=1.0), dict(temperature=0.7, top_k=40),
              dict(temperature=1.3, top_p=0.9), dict(temperature=0.8, top_k=50, top_p=0.95),
              dict(temperature=1.0, min_p=0.05), dict(temperature=0.9, min_p=0.02, top_k=20, top_p=0.8),
              dict(temperature=2.0, top_k=1), dict(temperature=1.0, top_k=5000), dict(temperature=1.0, top_p=0.3)]
    rows = 4 * len(combos)
    logits = rng.normal(0, 3, size=(rows, vocab)).astype(np.float32)
    logits[3] = np.round(logits[3])              # heavy ties
    logits[5] = np.round(logits[5] * 2) / 2
    logits[7, ::3] = -np.inf
    words = (vocab + 31) // 32
    masks = rng.integers(0, 2 ** 32, size=(3, words), dtype=np.uint64).astype(np.uint32)
    masks[1] &= rng.integers(0, 2 ** 32, size=words, dtype=np.uint64).astype(np.uint32)
    masks[2] = 0
    masks[2, 5] = 0b1011                         # three candidates only
    params = []
    for r in range(rows):
        c = combos[r % len(combos)]
        params.append(RowParams(seed=1234 + r, position=r * 7, mask_row=[-1, 0, 1, 2][r // len(combos)], **c))
    dev = torch.device("cuda")
    tok, st = sample_rows(torch.from_numpy(logits).to(dev), pack_params(params, dev),
                          torch.from_numpy(masks.view(np.int32)).to(dev))
    tok2, _ = sample_rows(torch.from_numpy(logits).to(dev), pack_params(params, dev),
                          torch.from_numpy(masks.view(np.int32)).to(dev))
    torch.cuda.synchronize()
    assert torch.equal(tok, tok2)
    tok, st = tok.cpu().numpy(), st.cpu().numpy()
    mismatches = 0
    for r, p in enumerate(params):
        m = masks[p.mask_row] if p.mask_row >= 0 else None
        want, err = _oracle(logits[r], m, p)
        assert (st[r] == 0) == (err == 0), (r, st[r], err)
        if err == 0 and tok[r] != want:
            mismatches += 1                      # only a draw that lands on a cumulative boundary may differ
    assert mismatches <= 1, mismatches


def test_sampler_statuses():
    from ds41rt_b200.ops.sampling import RowParams, pack_params, sample_rows
    dev = torch.device("cuda")
    vocab = 512
    logits = torch.randn(5, vocab, device=dev)
    logits[1, 7] = float("nan")
    logits[2, 9] = float("inf")
    masks = torch.zeros(1, vocab // 32, dtype=torch.int32, device=dev)
    params = [RowParams(temperature=-1.0), RowParams(temperature=0.0), RowParams(temperature=1.0),
              RowParams(temperature=1.0, mask_row=0), RowParams(temperature=1.0, top_p=0.0)]
    tok, st = sample_rows(logits, pack_params(params, dev), masks)
    assert st.tolist() == [3, 2, 2, 1, 6]


def test_sampler_adversarial_rows_match_host_oracle():
    """Rows built to sit on the sampler's decision boundaries (ideas from the reference's selftest,
    native/tests/v41_sampling_selftest.cu): ties straddling the top-k cut, k beyond the in-register selection width,
    all-equal rows, one dominant token, scaled values that fall into the subnormal range, huge negative logits, a
    single allowed token, an empty mask, min_p = 1, top_p at a cumulative boundary, near-greedy temperatures and a
    vocabulary that is not a multiple of 32.  Every row is drawn with four seeds and must equal the host oracle's
    token (or its error)."""
    from ds41rt_b200.ops.sampling import RowParams, pack_params, sample_rows
    rng = np.random.default_rng(7)
    vocab = 5003                                     # not a multiple of 32: the last mask word is partial
    words = (vocab + 31) // 32
    base = rng.normal(0, 2, size=vocab).astype(np.float32)
    rows, params = [], []

    def add(logit_row, mask_row=-1, **kw):
        for s in range(4):
            rows.append(np.asarray(logit_row, dtype=np.float32))
            params.append(RowParams(seed=99 + 17 * s + len(rows), position=3 * len(rows) + s, mask_row=mask_row, **kw))

    tie = base.copy()
    tie[100:160] = 5.0                               # 60 equal values on top: every cut below 60 splits the tie
    for k in (1, 7, 40, 59, 60, 61):
        add(tie, temperature=1.0, top_k=k)
    add(tie, temperature=0.7, top_k=50, top_p=0.5)
    for k in (256, 257, 300, 1000, vocab, vocab + 10):       # selection width boundary and no-op widths
        add(base, temperature=1.0, top_k=k)
    add(np.zeros(vocab), temperature=1.0)                     # all equal
    add(np.zeros(vocab), temperature=1.0, top_k=33, top_p=0.9)
    peak = base.copy()
    peak[4321] = 80.0                                        # one dominant token: everything else underflows
    add(peak, temperature=1.0)
    add(peak, temperature=1.0, top_p=0.999)
    add(base * 1e-30, temperature=2.0)                       # scaled differences are subnormal
    add(base * 1e-38, temperature=1.0, top_k=10)
    neg = base.copy()
    neg[::2] = -1e30                                         # finite but astronomically unlikely
    add(neg, temperature=1.0, top_p=0.95)
    add(base, temperature=1.0, min_p=1.0)                    # only the maxima survive
    add(tie, temperature=1.0, min_p=1.0)
    two = np.full(vocab, -50.0, dtype=np.float32)
    two[10], two[20] = 0.0, 0.0                              # two tokens at 0.5 each: top_p = 0.5 sits on the boundary
    add(two, temperature=1.0, top_p=0.5)
    add(two, temperature=1.0, top_p=0.5000001)
    for t in (1e-6, 9e-6, 1.1e-5, 1e-4, 1e-3):               # around the greedy threshold
        add(base, temperature=t)
    masks = np.zeros((3, words), dtype=np.uint32)
    masks[0, words - 1] = 1 << ((vocab - 1) % 32)            # only the last token of the vocabulary
    masks[1] = 0                                             # nothing allowed
    masks[2] = rng.integers(0, 2 ** 32, size=words, dtype=np.uint64).astype(np.uint32)
    masks[2, words - 1] &= (1 << (vocab % 32)) - 1
    add(base, mask_row=0, temperature=1.0, top_k=5)
    add(base, mask_row=0, temperature=0.0)
    add(base, mask_row=1, temperature=1.0)
    add(tie, mask_row=2, temperature=1.0, top_k=30)
    add(tie, mask_row=2, temperature=0.0)                    # masked greedy with ties: lowest allowed id
    logits = np.stack(rows)
    dev = torch.device("cuda")
    tok, st = sample_rows(torch.from_numpy(logits).to(dev), pack_params(params, dev),
                          torch.from_numpy(masks.view(np.int32)).to(dev))
    torch.cuda.synchronize()
    tok, st = tok.cpu().numpy(), st.cpu().numpy()
    bad = []
    for r, p in enumerate(params):
        m = masks[p.mask_row] if p.mask_row >= 0 else None
        want, err = _oracle(logits[r], m, p)
        if (st[r] == 0) != (err == 0) or (err == 0 and tok[r] != want):
            bad.append((r, int(st[r]), int(tok[r]), want, err))
    assert not bad, bad[:8]


def _tokens_at_the_draw(logits, mask, p):
    """Tokens that the draw may give when cumulative weights carry the rounding of the sums: a device weight is a whole number of
    2^-40 (half of one off), the oracle adds n of them in 64 bits."""
    from ds41rt_b200.runtime import core
    ids = np.arange(len(logits))
    if mask is not None:
        ids = ids[(mask[ids >> 5] >> (ids & 31).astype(np.uint32)) & 1 != 0]
    inv = np.float32(1) / np.float32(p.temperature)
    s = logits[ids] * inv
    top = s.max()
    if p.min_p > 0:
        keep = s >= np.float32(top + np.float32(np.log(np.float32(p.min_p))))
        ids, s = ids[keep], s[keep]
    if p.top_k > 0 or p.top_p < 1:
        order = np.lexsort((ids, -s.astype(np.float64)))
        order = order[:p.top_k] if p.top_k > 0 else order
        ids, s = ids[order], s[order]
    run = np.cumsum(np.exp(s.astype(np.float64) - np.float64(top)))
    n, total = len(run), run[-1]
    tol = n * 2.0 ** -40 + total * n * 2.0 ** -52
    at = lambda x: min(int(np.searchsorted(run, x)), n - 1)
    cut = float(np.float32(p.top_p)) * total
    ends = range(at(cut - tol), at(cut + tol) + 1) if p.top_p < 1 else [n - 1]
    u = float(core.sample_uniform(p.seed, p.position))
    return {int(ids[min(i, e)]) for e in ends for i in range(at(u * run[e] - 2 * tol), at(u * run[e] + 2 * tol) + 1)}


def test_tokens_at_the_draw_hold_the_oracles_token():
    """The bound's own check: nearly always one token, always the oracle's."""
    from ds41rt_b200.ops.sampling import RowParams
    rng = np.random.default_rng(3)
    single = 0
    for i in range(200):
        vocab = int(rng.integers(2, 3000))
        row = rng.normal(0, 2, size=vocab).astype(np.float32)
        kw = [dict(), dict(top_p=0.8), dict(top_k=7), dict(min_p=0.1), dict(top_k=20, top_p=0.9)][i % 5]
        p = RowParams(seed=i, position=3 * i, temperature=0.5 + 0.01 * i, **kw)
        got = _tokens_at_the_draw(row, None, p)
        assert _oracle(row, None, p)[0] in got
        single += len(got) == 1
    assert single >= 198


@pytest.mark.parametrize("vocab,offset", [(3, 0), (31, 1), (257, 3), (8 * 32 + 1, 0), (20011, 1), (8 * 49152 + 5, 0),
                                          ((8 << 18) + 3, 0)])
def test_sampler_slices_of_a_row(vocab, offset):
    """Where a row's slices are empty, short, unaligned or longer than a CTA's shared memory.  The draw takes integer weights, so
    a token may differ from the oracle's only where the draw lands on a boundary between two tokens (and never when greedy)."""
    from ds41rt_b200.ops.sampling import RowParams, pack_params, sample_rows
    rng = np.random.default_rng(vocab)
    asked = [dict(temperature=0.0), dict(temperature=1.0), dict(temperature=0.7, top_p=0.8), dict(temperature=0.9, top_k=7),
             dict(temperature=1.1, min_p=0.1), dict(temperature=1.0, top_k=2, top_p=0.9)]
    flat = rng.normal(0, 2, size=len(asked) * vocab + offset).astype(np.float32)
    flat[offset + vocab:offset + 2 * vocab] = 0.0            # all equal
    dev = torch.device("cuda")
    logits = torch.from_numpy(flat).to(dev)[offset:].view(len(asked), vocab)
    words = (vocab + 31) // 32
    masks = rng.integers(0, 2 ** 32, size=(1, words), dtype=np.uint64).astype(np.uint32)
    masks[0, 0] |= 2
    for mask_row in (-1, 0):
        params = [RowParams(seed=5 + i, position=i, mask_row=mask_row, **a) for i, a in enumerate(asked)]
        tok, st = sample_rows(logits, pack_params(params, dev), torch.from_numpy(masks.view(np.int32)).to(dev))
        for r, p in enumerate(params):
            row, mask = flat[offset + r * vocab:offset + (r + 1) * vocab], masks[0] if mask_row == 0 else None
            want, err = _oracle(row, mask, p)
            assert (int(st[r]) == 0) == (err == 0)
            if err == 0 and int(tok[r]) != want:
                assert p.temperature > 0 and {int(tok[r]), want} <= _tokens_at_the_draw(row, mask, p), (r, int(tok[r]), want)


@pytest.mark.parametrize("vocab,counts", [(4096, (8,)), (4097, (36, 37, 75)), (20000, (15, 16, 37, 74, 75, 150)), (40000, (24, 25, 75)),
                                          (60000, (40, 41, 101)), (100000, (64, 65))])
def test_a_row_gets_its_token_whatever_is_sampled_beside_it(vocab, counts):
    """How many CTAs share a row follows the number of rows and their length; sums are whole numbers, so the token does not."""
    from ds41rt_b200.ops.sampling import RowParams, pack_params, sample_rows
    rng = np.random.default_rng(vocab)
    asked = [dict(temperature=0.0), dict(temperature=1.0), dict(temperature=0.7, top_p=0.8), dict(temperature=0.9, top_k=7),
             dict(temperature=1.1, min_p=0.1), dict(temperature=1.0, top_k=2000, top_p=0.95), dict(temperature=1.4, top_p=0.999)]
    n = max(counts)
    dev = torch.device("cuda")
    logits = torch.from_numpy(rng.normal(0, 2, size=(n, vocab)).astype(np.float32)).to(dev)
    logits[1] = 0.0                                          # all equal
    logits[2, ::2] = 3.0
    masks = torch.from_numpy(rng.integers(0, 2 ** 32, size=(1, (vocab + 31) // 32), dtype=np.uint64).astype(np.uint32).view(np.int32)).to(dev)
    rows = [RowParams(seed=5 + i, position=i, mask_row=0 if i % 3 == 2 else -1, **asked[i % len(asked)]) for i in range(n)]
    alone = [sample_rows(logits[i:i + 1], pack_params([rows[i]], dev), masks) for i in range(n)]
    tok, st = (torch.cat([a[j] for a in alone]) for j in (0, 1))
    assert not bool(st.any())
    for m in counts:
        t, s = sample_rows(logits[:m], pack_params(rows[:m], dev), masks)
        assert torch.equal(t, tok[:m]) and not bool(s.any())


@pytest.mark.parametrize("ties", [False, True])
@pytest.mark.parametrize("members", [1, 2, 31, 94, 95, 96, 97, 98, 200, 510, 511, 600])
def test_gathered_lists_of_any_length(members, ties):
    """All that a selection has to tell apart in one bin of its histogram, around the length where a list is searched by lanes together."""
    from ds41rt_b200.ops.sampling import RowParams, pack_params, sample_rows
    rng = np.random.default_rng(members)
    vocab, dev = 6000, torch.device("cuda")
    row = rng.normal(-12, 1, size=vocab).astype(np.float32)
    at = rng.choice(vocab, members, replace=False)
    row[at] = 2.0 - (rng.integers(0, 7, members) / 256 if ties else rng.permutation(members) / (members * 40.0))
    asked = [dict(top_k=max(1, members // 2)), dict(top_p=0.5), dict(top_p=0.97), dict(top_k=members, top_p=0.3), dict(min_p=0.5, top_p=0.8),
             dict(top_k=members + 3), dict()]
    rows = [RowParams(temperature=1.0, seed=s, position=s, **asked[s % len(asked)]) for s in range(4 * len(asked))]
    logits = torch.from_numpy(row).to(dev).expand(len(rows), vocab).contiguous()
    tok, st = sample_rows(logits, pack_params(rows, dev))
    assert not bool(st.any())
    for r, p in enumerate(rows):
        want, _ = _oracle(row, None, p)
        if int(tok[r]) != want:
            assert {int(tok[r]), want} <= _tokens_at_the_draw(row, None, p), (r, int(tok[r]), want)

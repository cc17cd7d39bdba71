"""Kernels that ask for a pass's cache rows before the wait for the previous kernel, when that kernel is the one that moves the
positions on (a loop on the device without a graph)."""
import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu


def _settled_and_late(call, pos, out):
    """Results of call() with the positions in place, and with the step that writes them still waiting when the call's blocks start:
    it stands behind a product of one block that takes milliseconds and lets its successors start at once."""
    from ds41rt_b200.ops import gemm as G, lib
    k, rows = lib.kernels(), pos.numel()
    got = []
    x, w = torch.ones(32, 1 << 18, device="cuda").bfloat16(), torch.ones(128, 1 << 18, device="cuda").bfloat16()
    y, st = torch.zeros(32, 128, device="cuda"), lib.new_status("cuda")
    chosen, tokens = torch.zeros(2, rows, dtype=torch.int32, device="cuda").unbind()
    long = lambda: G.gemm_raw(w, x, y, 128, 32, 1 << 18, lda=1 << 18, ldb=1 << 18, ldo=128, out_mode=3, bn=32, status=st)
    long()
    for late in (False, True):
        for t in out:
            t.zero_()
        before = pos.clone()
        if late:
            pos -= 1
        torch.cuda.synchronize()
        if late:
            long()
            lib.check(k.ds41_decode_feedback(lib.ptr(chosen), lib.ptr(tokens), lib.ptr(pos), rows, lib.stream()), "feedback")
        call()
        torch.cuda.synchronize()
        assert torch.equal(pos, before)
        got.append([t.clone() for t in out])
    lib.raise_on_status(st, "late positions")
    assert all(bool(t.any()) for t in got[0])
    for a, b in zip(*got):
        assert torch.equal(a, b)


def _paged(slots, pages, page, row_len):
    g = torch.Generator().manual_seed(pages)
    table = torch.randperm(slots * pages, generator=g).int().view(slots, pages).cuda()
    return table, torch.randn((slots * pages + 1) * page, row_len, generator=g).bfloat16().cuda()


# positions that move on to a new tile of 64 keys, to a new page, into a new split's share
POSITIONS = [[64], [128, 63, 640], [1, 959]]


@pytest.mark.parametrize("positions", POSITIONS)
@pytest.mark.parametrize("heads,kv", [(16, 512), (32, 512), (8, 128)])
def test_latent_attention(heads, kv, positions):
    from ds41rt_b200.ops import lib, stack as S
    rows, splits, rot, page = len(positions), 8, 64, 64
    table, pool = _paged(rows, 16, page, kv + rot)
    q = torch.randn(rows, heads * (kv + rot), device="cuda").bfloat16() * 0.2
    pos, slot = torch.tensor(positions, dtype=torch.int32).cuda(), torch.arange(rows, dtype=torch.int32).cuda()
    part, ml, st = torch.zeros(rows, splits, heads, kv).cuda(), torch.zeros(rows, splits, heads, 2).cuda(), lib.new_status("cuda")
    a = S.LatentAttendArgs()
    a.q_abs, a.q_rot, a.pool, a.page_table, a.row_pos, a.row_slot, a.part_o, a.part_ml, a.status = (
        lib.ptr(t) for t in (q, q[:, heads * kv:], pool, table, pos, slot, part, ml, st))
    a.ld_q_abs, a.ld_q_rot, a.q_rot_stride, a.scale, a.rows, a.heads = q.shape[1], q.shape[1], rot, 0.05, rows, heads
    a.kv_pad, a.row_len, a.n_splits, a.max_pages, a.page_tokens = kv, kv + rot, splits, table.shape[1], page
    _settled_and_late(lambda: lib.check(lib.kernels().ds41_latent_attend(C.byref(a), lib.stream()), "attend"), pos, [part, ml])
    lib.raise_on_status(st, "latent")


@pytest.mark.parametrize("positions", POSITIONS)
@pytest.mark.parametrize("heads,groups,dim,chunk", [(16, 4, 128, 0), (8, 8, 64, 128)])
def test_grouped_attention(heads, groups, dim, chunk, positions):
    from ds41rt_b200.ops import lib, stack as S
    rows, page = len(positions), 64
    table, pool = _paged(rows, 16, page, groups * 2 * dim)
    q = torch.randn(rows, heads * dim, device="cuda").bfloat16()
    pos, slot = torch.tensor(positions, dtype=torch.int32).cuda(), torch.arange(rows, dtype=torch.int32).cuda()
    out, st = torch.zeros(rows, heads * dim, device="cuda").bfloat16(), lib.new_status("cuda")
    a = S.GroupAttendArgs()
    a.q, a.pool, a.page_table, a.row_pos, a.row_slot, a.out, a.status = (lib.ptr(t) for t in (q, pool, table, pos, slot, out, st))
    a.gate, a.u, a.ld_q, a.scale = S.NO_PROJ, S.NO_PROJ, heads * dim, dim ** -0.5
    a.rows, a.heads, a.kv_heads, a.dim_pad, a.vdim_pad, a.chunk = rows, heads, groups, dim, dim, chunk
    a.taps, a.slots, a.n_splits, a.ld_out, a.max_pages = 1, rows, 4, heads * dim, table.shape[1]
    a.page_tokens, a.n_pages = page, rows * 16
    _settled_and_late(lambda: lib.check(lib.kernels().ds41_group_attend(C.byref(a), lib.stream()), "attend"), pos, [out])
    lib.raise_on_status(st, "grouped")


@pytest.mark.parametrize("positions", POSITIONS)
@pytest.mark.parametrize("D,heads,rope", [(512, 64, 64), (128, 8, 32)])
def test_window_attention(D, heads, rope, positions):
    """The rotation's table is made before the wait, too."""
    from ds41rt_b200.config import RopeConfig, rope_inv_freq
    from ds41rt_b200.ops import attention as A, lib
    rows, window, ring, splits = len(positions), 128, 144, 3
    win = torch.randn(rows, ring, D, device="cuda").bfloat16()
    q, sink = torch.randn(rows, heads * D, device="cuda").bfloat16(), torch.randn(heads, device="cuda")
    pos, slot = torch.tensor(positions, dtype=torch.int32).cuda(), torch.arange(rows, dtype=torch.int32).cuda()
    part_o, part_ml = torch.zeros(rows, splits, heads, D, device="cuda"), torch.zeros(rows, splits, heads, 2, device="cuda")
    out = torch.zeros(rows, heads * D, device="cuda").bfloat16()
    sel, none = torch.full((rows, 16), -1, dtype=torch.int32, device="cuda"), torch.zeros(rows, dtype=torch.int32, device="cuda")
    table = torch.zeros(rows, 1, dtype=torch.int32, device="cuda")
    inv = torch.tensor(rope_inv_freq(RopeConfig(), rope), device="cuda")
    call = lambda: lib.check(A.attend(q=q, ldq=heads * D, q_off=0, rows=rows, heads=heads, D=D, window=window, ring=ring, row_pos=pos,
                                      row_slot=slot, win=win, comp_pool=None, sel=sel, n_sel=none, k=16, page_table=table,
                                      max_pages=1, page_rows=1, inv_freq=inv, rope_dim=rope, scale=D ** -0.5, n_splits=splits,
                                      part_o=part_o, part_ml=part_ml, sink=sink, out=out, ldo=heads * D, impl="legacy"), "attend")
    _settled_and_late(call, pos, [out])

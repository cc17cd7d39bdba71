"""Individual CUDA kernels vs plain PyTorch fp32 references of the same op."""
import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("max_keys,positions", [(5000, [4999, 2999, 300, 4000]),        # register forms (8 / 4 keys a thread)
                                                (20000, [15999, 19999, 2047, 9000]),    # 16 a thread; streaming form
                                                (1024, [1023, 700, 511, 600])])
def test_topk_select_exact(max_keys, positions):
    from ds41rt_b200.ops import lib
    k = lib.kernels()
    rows, topk = 4, 512
    torch.manual_seed(0)
    scores = torch.randn(rows, max_keys, device="cuda")
    scores[1, :3000] = scores[1, :3000].round()            # many ties
    scores[0, 17] = float("-inf")
    pos = torch.tensor(positions, dtype=torch.int32, device="cuda")
    slot = torch.tensor([0, 0, 0, -1], dtype=torch.int32, device="cuda")
    sel = torch.zeros(rows, topk, dtype=torch.int32, device="cuda")
    n_sel = torch.zeros(rows, dtype=torch.int32, device="cuda")
    lib.check(k.ds41_topk_select(lib.ptr(scores), max_keys, lib.ptr(pos), lib.ptr(slot), 1, topk, lib.ptr(sel),
                                 lib.ptr(n_sel), rows, lib.stream()), "topk")
    torch.cuda.synchronize()
    for r in range(3):
        n = int(pos[r]) + 1
        got = sel[r, : int(n_sel[r])].tolist()
        if n <= topk:
            assert got == list(range(n))
            continue
        s = scores[r, :n].cpu()
        order = torch.sort(s, descending=True, stable=True).indices[:topk]
        assert got == sorted(order.tolist())
        assert int(n_sel[r]) == topk
    assert int(n_sel[3]) == 0


@pytest.mark.parametrize("masked", [False, True])
@pytest.mark.parametrize("max_keys,ratio", [(513, 1), (2048, 1), (2049, 1), (4097, 1), (8192, 1), (16000, 2)])
def test_topk_of_many_rows(max_keys, ratio, masked):
    """Passes of many rows choose what passes of few rows choose (which the test above compares with a sort)."""
    from ds41rt_b200.ops import lib
    k = lib.kernels()
    rows, topk, block = 400, 512, 8
    torch.manual_seed(max_keys)
    scores = torch.randn(rows, max_keys, device="cuda")
    scores[::3] = scores[::3].round()                      # many ties
    scores[1] = float("-inf")
    scores[2, ::2] = float("inf")
    pos = torch.randint(0, ratio * max_keys + 5, (rows,), device="cuda", dtype=torch.int32)
    pos[3:6] = torch.tensor([ratio * max_keys - 1, 511, 512], dtype=torch.int32)
    slot = torch.where(torch.arange(rows, device="cuda") % 50 == 7, -1, 0).int()
    words = (max_keys + 32 * block - 1) // (32 * block)
    mask = torch.randint(-2 ** 31, 2 ** 31, (rows, words), device="cuda", dtype=torch.int64).int()
    got = []
    for step in (rows, 100):
        sel, n_sel = torch.zeros(rows, topk, dtype=torch.int32, device="cuda"), torch.zeros(rows, dtype=torch.int32, device="cuda")
        for r in range(0, rows, step):
            lib.check(k.ds41_topk_select_cand(lib.ptr(scores[r:]), max_keys, lib.ptr(pos[r:]), lib.ptr(slot[r:]), ratio, topk,
                                              lib.ptr(sel[r:]), lib.ptr(n_sel[r:]), step, lib.ptr(mask[r:]) if masked else None,
                                              words if masked else 0, block if masked else 0, lib.stream()), "topk")
        torch.cuda.synchronize()
        got.append((sel, n_sel))
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])
    assert masked or int(got[0][1].max()) == topk          # a mask of random bits leaves half of the keys


@pytest.mark.parametrize("rows", [296, 297, 592, 593])
@pytest.mark.parametrize("keys", [4096, 5120, 5121, 8192, 8193])
def test_topk_around_the_lines_of_its_forms(rows, keys):
    """The rows of a long pass choose what each of them chooses in a pass of few."""
    from ds41rt_b200.ops import lib
    k, topk = lib.kernels(), 512
    torch.manual_seed(keys + rows)
    scores = torch.randn(rows, keys, device="cuda")
    scores[::2] = (scores[::2] * 4).round()
    pos = torch.randint(0, keys, (rows,), device="cuda", dtype=torch.int32)
    pos[::3] = keys - 1
    slot = torch.zeros(rows, dtype=torch.int32, device="cuda")
    got = []
    for step in (rows, 74):
        sel, n = torch.zeros(rows, topk, dtype=torch.int32, device="cuda"), torch.zeros(rows, dtype=torch.int32, device="cuda")
        for r in range(0, rows, step):
            lib.check(k.ds41_topk_select(lib.ptr(scores[r:]), keys, lib.ptr(pos[r:]), lib.ptr(slot[r:]), 1, topk, lib.ptr(sel[r:]),
                                         lib.ptr(n[r:]), min(step, rows - r), lib.stream()), "topk")
        torch.cuda.synchronize()
        got.append((sel, n))
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])


def _attend_ref(q, keys, sink, scale):
    # q [H, D], keys [n, D]
    logits = (q @ keys.t()) * scale
    m = torch.maximum(logits.amax(-1, keepdim=True), sink[:, None])
    e = torch.exp(logits - m)
    return (e / (e.sum(-1, keepdim=True) + torch.exp(sink[:, None] - m))) @ keys


def _pack_fp8_rows(x, row_bytes):
    """bf16 rows -> (FP8 cache rows [.., row_bytes] uint8, the dequantised values the kernel must see)."""
    from ds41rt_b200.ops import quant_ref as Q
    D = x.shape[-1]
    q, e = Q.quant_mxfp8(x.float(), 32)
    rows = torch.zeros(*x.shape[:-1], row_bytes, dtype=torch.uint8, device=x.device)
    rows[..., :D] = q.view(torch.uint8)
    rows[..., D:D + D // 32] = e.to(torch.uint8)
    return rows.contiguous(), Q.dequant_mxfp8(q, e, 32).bfloat16()


def _pack_fp4_rows(x, row_bytes):
    """bf16 rows -> (FP4 cache rows [.., row_bytes] uint8, the dequantised values the kernel must see)."""
    from ds41rt_b200.ops import quant_ref as Q
    D = x.shape[-1]
    packed, bs = Q.quant_kv_fp4_e4m3_16(x.float())
    rows = torch.zeros(*x.shape[:-1], row_bytes, dtype=torch.uint8, device=x.device)
    rows[..., :D // 2] = packed.view(torch.uint8).reshape(*x.shape[:-1], D // 2)
    rows[..., D // 2:D // 2 + D // 16] = bs.view(torch.uint8).reshape(*x.shape[:-1], D // 16)
    return rows.contiguous(), Q.dequant_kv_fp4_e4m3_16(packed, bs).reshape(x.shape).bfloat16()


@pytest.mark.parametrize("impl", ["tc", "legacy"])
@pytest.mark.parametrize("kv", ["bf16", "fp8", "fp4"])
@pytest.mark.parametrize("D,heads,rope,rows,n_splits", [(128, 8, 32, 3, 0), (512, 16, 64, 3, 0), (512, 64, 64, 3, 0),
                                                         (512, 64, 64, 70, 1), (512, 64, 64, 66, 3), (128, 64, 32, 64, 2),
                                                         (512, 64, 64, 330, 1), (512, 8, 64, 180, 2)])
def test_sparse_attention(D, heads, rope, rows, n_splits, kv, impl):
    """impl "tc": tcgen05 kernel (persistent grid over (row, key split) items, accumulators in tensor memory, final rows
    written by the kernel when there is one split); "legacy": warp-MMA kernels (rows >= 64 with 64 heads runs their wide
    form)."""
    from ds41rt_b200.ops import lib
    from ds41rt_b200.ops import attention as A
    from ds41rt_b200.config import RopeConfig, rope_inv_freq
    from ds41rt_b200.models.reference import apply_rope
    k = lib.kernels()
    torch.manual_seed(0)
    window, ring, topk, page_rows, max_pages = 128, 144 + rows, 64, 32, 16
    positions = ([700, 701, 50] + [300 + 3 * i for i in range(rows)])[:rows]
    slots = ([0, 0, 1] + [i % 2 for i in range(rows)])[:rows]
    win = torch.randn(2, ring, D, device="cuda").bfloat16()
    pool = torch.randn(max_pages * 2 * page_rows, D, device="cuda").bfloat16()
    row_bytes = 0 if kv == "bf16" else (D + D // 32 + 15) // 16 * 16      # "fp4" keeps FP8 window rows
    win_dev, pool_dev = win, pool
    comp_bytes = 0
    if row_bytes:
        win_dev, win = _pack_fp8_rows(win, row_bytes)          # the reference below sees the dequantised rows
        if kv == "fp4":                                        # FP8 window rows, FP4 compressed rows
            comp_bytes = (D // 2 + D // 16 + 15) // 16 * 16
            pool_dev, pool = _pack_fp4_rows(pool, comp_bytes)
        else:
            pool_dev, pool = _pack_fp8_rows(pool, row_bytes)
    page_table = torch.arange(2 * max_pages, dtype=torch.int32, device="cuda").view(2, max_pages).flip(1).contiguous()
    sel = torch.full((rows, topk), -1, dtype=torch.int32, device="cuda")
    counts = ([64, 40, 0] + [(7 * i) % 65 for i in range(rows)])[:rows]
    n_sel = torch.tensor(counts, dtype=torch.int32, device="cuda")
    for i, c in enumerate(counts):
        if c:
            sel[i, :c] = torch.sort(torch.randperm(300)[:c]).values.int().cuda()
    q = torch.randn(rows, heads * D, device="cuda").bfloat16()
    sink = torch.randn(heads, device="cuda")
    inv = torch.tensor(rope_inv_freq(RopeConfig(), rope), device="cuda")
    n_splits = n_splits or (window + 16 + topk + 63) // 64
    part_o = torch.zeros(rows, n_splits, heads, D, device="cuda")
    part_ml = torch.zeros(rows, n_splits, heads, 2, device="cuda")
    out = torch.zeros(rows, heads * D, device="cuda", dtype=torch.bfloat16)
    pos_t = torch.tensor(positions, dtype=torch.int32, device="cuda")
    slot_t = torch.tensor(slots, dtype=torch.int32, device="cuda")
    scale = D ** -0.5
    status = lib.new_status(q.device)
    lib.check(A.attend(q=q, ldq=heads * D, q_off=0, rows=rows, heads=heads, D=D, window=window, ring=ring, row_pos=pos_t,
                       row_slot=slot_t, win=win_dev, comp_pool=pool_dev, sel=sel, n_sel=n_sel, k=topk,
                       page_table=page_table, max_pages=max_pages, page_rows=page_rows, inv_freq=inv, rope_dim=rope,
                       scale=scale, n_splits=n_splits, part_o=part_o, part_ml=part_ml, sink=sink, out=out,
                       ldo=heads * D, kv_row_bytes=row_bytes, comp_row_bytes=comp_bytes, status=status, impl=impl),
              "attend")
    torch.cuda.synchronize()
    lib.raise_on_status(status, "attend")
    torch.cuda.synchronize()
    for r in range(rows):
        pos, slot = positions[r], slots[r]
        lo = max(0, pos - window + 1)
        keys = [win[slot, p % ring] for p in range(lo, pos + 1)]
        for j in range(int(n_sel[r])):
            i = int(sel[r, j])
            phys = int(page_table[slot, i // page_rows]) * page_rows + i % page_rows
            keys.append(pool[phys])
        keys = torch.stack(keys).float()
        qr = apply_rope(q[r].float().view(heads, D).cpu(), torch.tensor(pos), inv.cpu(), rope).cuda()
        qr = qr.bfloat16().float()
        want = _attend_ref(qr, keys, sink, scale)
        want = apply_rope(want.cpu(), torch.tensor(pos), inv.cpu(), rope, inverse=True).cuda()
        got = out[r].float().view(heads, D)
        err = float((got - want).abs().max())
        assert err < 3e-2 * float(want.abs().max()) + 2e-3, (r, err)


def test_hc_kernels_match_oracle():
    from ds41rt_b200.ops import lib
    from ds41rt_b200.models import reference as R
    k = lib.kernels()
    torch.manual_seed(0)
    rows, H = 5, 512
    streams = torch.randn(rows, 4, H, device="cuda").bfloat16()
    sub = torch.randn(2, rows, H, device="cuda")           # two split planes
    fn = torch.randn(24, 4 * H, device="cuda") * 0.5
    scale = torch.tensor([1.0, 0.7, 1.3], device="cuda")
    base = torch.randn(24, device="cuda") * 0.5
    pre_in = torch.rand(rows, 4, device="cuda")
    norm_w = torch.rand(H, device="cuda") + 0.5
    # reference: mixes on the ORIGINAL streams give post/comb for the expand
    pre0, post0, comb0 = R.hc_mixes(streams.float().cpu(), fn.cpu(), scale.cpu(), base.cpu(), 4, 20, 1e-6, 1e-20)
    subsum = sub.sum(0).bfloat16().float().cpu()
    new_streams = R.hc_expand(streams.float().cpu(), subsum, post0, comb0).bfloat16().float()
    pre1, post1, comb1 = R.hc_mixes(new_streams, fn.cpu(), scale.cpu(), base.cpu(), 4, 20, 1e-6, 1e-20)
    xn = R.rmsnorm(R.hc_collapse(new_streams, pre_in.cpu()), norm_w.cpu(), 1e-20)
    # kernels
    st = lib.new_status("cuda")
    s_dev = streams.clone()
    partial = torch.zeros(H // 128, rows, 25, device="cuda")
    bases = (C.c_void_p * 1)(sub.data_ptr())
    post_d, comb_d = post0.cuda().contiguous(), comb0.reshape(rows, 16).cuda().contiguous()
    lib.check(k.ds41_hc_post_mix(lib.ptr(s_dev), lib.ptr(s_dev), bases, 1, 2, C.c_longlong(rows * H), lib.ptr(post_d),
                                 lib.ptr(comb_d), lib.ptr(fn), lib.ptr(partial), rows, H, lib.ptr(None), lib.ptr(None),
                                 lib.ptr(st), lib.ptr(None), lib.ptr(None), lib.ptr(None), lib.ptr(None), C.c_float(0.0), lib.stream()), "post_mix")
    next_pre = torch.zeros(rows, 4, device="cuda")
    post = torch.zeros(rows, 4, device="cuda")
    comb = torch.zeros(rows, 16, device="cuda")
    xn_d = torch.zeros(rows, H, device="cuda", dtype=torch.bfloat16)
    lib.check(k.ds41_hc_finish(lib.ptr(partial), H // 128, lib.ptr(scale), lib.ptr(base), lib.ptr(pre_in),
                               lib.ptr(s_dev), lib.ptr(norm_w), lib.ptr(next_pre), lib.ptr(post), lib.ptr(comb),
                               lib.ptr(xn_d), lib.ptr(None), lib.ptr(None), lib.ptr(None), rows, H, 20, C.c_float(1e-6), C.c_float(1e-20),
                               lib.ptr(None), 0, C.c_longlong(0), 0, lib.stream()), "finish")
    torch.cuda.synchronize()
    assert (s_dev.float().cpu() - new_streams).abs().max() < 0.05
    assert (next_pre.cpu() - pre1).abs().max() < 2e-2
    assert (post.cpu() - post1).abs().max() < 2e-2
    assert (comb.cpu().view(rows, 4, 4) - comb1).abs().max() < 2e-2
    assert (xn_d.float().cpu() - xn).abs().max() < 5e-2


def test_router_select_and_plan():
    from ds41rt_b200.ops import lib
    from ds41rt_b200.models import reference as R
    k = lib.kernels()
    torch.manual_seed(0)
    rows, E, I_sh, topk = 6, 384, 64, 6
    planes = torch.randn(2, rows, E + 2 * I_sh, device="cuda")
    bias = torch.randn(E, device="cuda") * 0.01
    ids = torch.zeros(rows, topk, dtype=torch.int32, device="cuda")
    wts = torch.zeros(rows, topk, device="cuda")
    act = torch.zeros(rows, I_sh, device="cuda", dtype=torch.bfloat16)
    lib.check(k.ds41_router_select(lib.ptr(planes), 2, rows, E + 2 * I_sh, E, I_sh, topk, lib.ptr(bias),
                                   C.c_float(1.5), C.c_float(10.0), lib.ptr(ids), lib.ptr(wts), lib.ptr(act),
                                   lib.stream()), "router")
    torch.cuda.synchronize()
    logits = planes.sum(0)[:, :E].cpu()
    score = torch.sqrt(torch.nn.functional.softplus(logits))
    order = torch.sort(score + bias.cpu(), dim=-1, descending=True, stable=True).indices[:, :topk]
    sel = torch.gather(score, 1, order)
    want_w = sel / sel.sum(-1, keepdim=True) * 1.5
    assert ids.cpu().tolist() == order.tolist()
    assert (wts.cpu() - want_w).abs().max() < 1e-5
    gsum = planes.sum(0).cpu()
    want_act = R.swiglu_clamped(gsum[:, E:E + I_sh].bfloat16().float(), gsum[:, E + I_sh:].bfloat16().float(), 10.0)
    assert (act.float().cpu() - want_act).abs().max() < 2e-2
    # plan for a rank owning experts [96, 192)
    slot = torch.zeros(rows, dtype=torch.int32, device="cuda")
    max_active = 36
    active = torch.zeros(max_active, dtype=torch.int32, device="cuda")
    n_active = torch.zeros(1, dtype=torch.int32, device="cuda")
    row_w = torch.zeros(max_active, 8, device="cuda")
    slot_of = torch.zeros(rows, topk, dtype=torch.int32, device="cuda")
    lib.check(k.ds41_moe_plan(lib.ptr(ids), lib.ptr(wts), lib.ptr(slot), rows, topk, 96, 192, max_active, 8,
                              lib.ptr(active), lib.ptr(n_active), lib.ptr(row_w), lib.ptr(slot_of), lib.stream()),
              "plan")
    torch.cuda.synchronize()
    local = sorted({int(e) - 96 for e in order.flatten().tolist() if 96 <= e < 192})
    assert int(n_active) == len(local)
    assert active[: len(local)].tolist() == local
    for r in range(rows):
        for j in range(topk):
            e = int(order[r, j])
            s = int(slot_of[r, j])
            if 96 <= e < 192:
                assert local[s] == e - 96 and abs(float(row_w[s, r]) - float(want_w[r, j])) < 1e-5
            else:
                assert s == -1


@pytest.mark.parametrize("group", [32, 128])
def test_act_quant_mx(group):
    from ds41rt_b200.ops import lib, quant_ref as Q
    from ds41rt_b200.ops.mx import unpack_sf_atoms
    k = lib.kernels()
    rows, K = 37, 512
    x = (torch.randn(rows, K, device="cuda") * torch.exp(torch.randn(rows, 1, device="cuda"))).bfloat16()
    q = torch.zeros(rows, K, dtype=torch.uint8, device="cuda")
    sf = torch.zeros(1, K // 128, 512, dtype=torch.uint8, device="cuda")
    lib.check(k.ds41_act_quant_mx(lib.ptr(x), C.c_longlong(K), C.c_longlong(0), lib.ptr(q), C.c_longlong(K),
                                  C.c_longlong(0), lib.ptr(sf), C.c_longlong(0), rows, K, 1, group, lib.ptr(None),
                                  lib.stream()), "act_quant")
    torch.cuda.synchronize()
    wq, we = Q.quant_act_fp8_ue8m0(x.float().cpu(), group)
    got_e = unpack_sf_atoms(sf.cpu(), rows)
    assert torch.equal(got_e, we)
    assert torch.equal(q.cpu().view(torch.float8_e4m3fn).float(), wq.float())


def test_hc_step_matches_unfused_kernels():
    """The fused hyper-connection step equals post_mix + finish run separately (same inputs)."""
    from ds41rt_b200.ops import lib
    k = lib.kernels()
    torch.manual_seed(1)
    rows, H = 3, 1024
    streams = torch.randn(rows, 4, H, device="cuda").bfloat16()
    sub = torch.randn(2, rows, H, device="cuda")
    fn = torch.randn(24, 4 * H, device="cuda") * 0.02
    scale = torch.tensor([1.0, 0.7, 1.3], device="cuda")
    base = torch.randn(24, device="cuda") * 0.5
    pre_in = torch.rand(rows, 4, device="cuda")
    post = torch.rand(rows, 4, device="cuda") * 2
    comb = torch.rand(rows, 16, device="cuda")
    norm_w = torch.rand(H, device="cuda") + 0.5
    st = lib.new_status("cuda")
    bases = (C.c_void_p * 1)(sub.data_ptr())
    # unfused
    s1 = streams.clone()
    partial = torch.zeros(H // 128, rows, 25, device="cuda")
    lib.check(k.ds41_hc_post_mix(lib.ptr(s1), lib.ptr(s1), bases, 1, 2, C.c_longlong(rows * H), lib.ptr(post),
                                 lib.ptr(comb), lib.ptr(fn), lib.ptr(partial), rows, H, lib.ptr(None), lib.ptr(None),
                                 lib.ptr(st), lib.ptr(None), lib.ptr(None), lib.ptr(None), lib.ptr(None), C.c_float(0.0), lib.stream()), "post_mix")
    np1, po1, co1 = torch.zeros(rows, 4, device="cuda"), torch.zeros(rows, 4, device="cuda"), torch.zeros(rows, 16, device="cuda")
    xn1 = torch.zeros(rows, H, device="cuda", dtype=torch.bfloat16)
    lib.check(k.ds41_hc_finish(lib.ptr(partial), H // 128, lib.ptr(scale), lib.ptr(base), lib.ptr(pre_in),
                               lib.ptr(s1), lib.ptr(norm_w), lib.ptr(np1), lib.ptr(po1), lib.ptr(co1), lib.ptr(xn1),
                               lib.ptr(None), lib.ptr(None), lib.ptr(None), rows, H, 20, C.c_float(1e-6),
                               C.c_float(1e-20), lib.ptr(None), 0, C.c_longlong(0), 0, lib.stream()), "finish")
    # fused (run twice: the ticket counters must reset themselves)
    for _ in range(2):
        s2 = streams.clone()
        a = lib.HcStepArgs()
        np2, po2, co2 = torch.zeros(rows, 4, device="cuda"), torch.zeros(rows, 4, device="cuda"), torch.zeros(rows, 16, device="cuda")
        xn2 = torch.zeros(rows, H, device="cuda", dtype=torch.bfloat16)
        xq = torch.zeros(rows, H, device="cuda", dtype=torch.uint8)
        xq_sf = torch.zeros(1, H // 128, 512, device="cuda", dtype=torch.uint8)
        if _ == 0:
            tickets = torch.zeros(rows, dtype=torch.int32, device="cuda")
        part2 = torch.zeros(H // 128, rows, 26, device="cuda")
        xc = torch.zeros(rows, H, device="cuda")
        a.streams_in = a.streams_out = lib.ptr(s2)
        a.part_bases = C.cast(bases, C.c_void_p)
        a.post, a.comb, a.pre_in = lib.ptr(post), lib.ptr(comb), lib.ptr(pre_in)
        a.fn, a.scale, a.base, a.norm_w = lib.ptr(fn), lib.ptr(scale), lib.ptr(base), lib.ptr(norm_w)
        a.partial, a.xc = lib.ptr(part2), lib.ptr(xc)
        a.next_pre, a.post_out, a.comb_out, a.xn = lib.ptr(np2), lib.ptr(po2), lib.ptr(co2), lib.ptr(xn2)
        a.xq, a.xq_sf, a.tickets, a.status = lib.ptr(xq), lib.ptr(xq_sf), lib.ptr(tickets), lib.ptr(st)
        a.split_stride, a.n_ranks, a.n_splits = rows * H, 1, 2
        a.rows, a.H, a.iters, a.hc_eps, a.norm_eps = rows, H, 20, 1e-6, 1e-20
        lib.check(k.ds41_hc_step(C.byref(a), lib.stream()), "hc_step")
        torch.cuda.synchronize()
        assert torch.equal(s1, s2)
        assert (np1 - np2).abs().max() < 1e-5 and (po1 - po2).abs().max() < 1e-5 and (co1 - co2).abs().max() < 1e-5
        assert (xn1.float() - xn2.float()).abs().max() < 2e-2
        assert int(tickets.abs().sum()) == 0
    from ds41rt_b200.ops import quant_ref as Q
    from ds41rt_b200.ops.mx import unpack_sf_atoms
    wq, we = Q.quant_act_fp8_ue8m0(xn2.float().cpu(), 128)
    assert torch.equal(unpack_sf_atoms(xq_sf.cpu(), rows), we)
    assert torch.equal(xq.cpu().view(torch.float8_e4m3fn).float(), wq.float())


def test_index_scores_on_tensor_cores_match_the_scalar_kernel():
    """One request, a long pass: RoPE'd queries x gathered keys as a GEMM with the relu / head-weight / head-sum
    epilogue gives the scores of the per-key kernel (same bf16 operands, fp32 accumulation)."""
    from ds41rt_b200.config import RopeConfig, rope_inv_freq
    from ds41rt_b200.ops import gemm as G, lib
    k = lib.kernels()
    torch.manual_seed(7)
    rows, IH, ID, ratio, page_rows, max_pages, max_keys = 200, 32, 128, 2, 32, 80, 2560
    pos0 = 3000
    positions = torch.arange(pos0, pos0 + rows, dtype=torch.int32, device="cuda")
    slots = torch.zeros(rows, dtype=torch.int32, device="cuda")
    ldq = IH * ID + 64
    q = torch.randn(rows, ldq, device="cuda").bfloat16()
    w_stride, w_off = 40, 8
    w = torch.randn(rows, w_stride, device="cuda")
    pool = torch.randn(max_pages * page_rows, ID, device="cuda").bfloat16()
    page_table = torch.randperm(max_pages, device="cuda").int().view(1, max_pages).contiguous()
    inv = torch.tensor(rope_inv_freq(RopeConfig(), ID // 2), device="cuda")
    ref = torch.full((rows, max_keys), float("nan"), device="cuda")
    lib.check(k.ds41_index_score(lib.ptr(q), C.c_longlong(ldq), 64, lib.ptr(w), w_stride, w_off, lib.ptr(pool),
                                 lib.ptr(page_table), max_pages, page_rows, lib.ptr(positions), lib.ptr(slots),
                                 lib.ptr(inv), rows, IH, ID, ratio, lib.ptr(ref), max_keys, lib.stream()), "score")
    n_keys = (pos0 + rows) // ratio
    qr = torch.zeros(rows * IH, ID, device="cuda", dtype=torch.bfloat16)
    kc = torch.zeros(max_keys, ID, device="cuda", dtype=torch.bfloat16)
    vis = torch.zeros(rows, dtype=torch.int32, device="cuda")
    got = torch.full((rows, max_keys), float("nan"), device="cuda")
    st = lib.new_status("cuda")
    lib.check(k.ds41_index_prepare(lib.ptr(q), C.c_longlong(ldq), 64, lib.ptr(pool), lib.ptr(page_table), max_pages,
                                   page_rows, lib.ptr(positions), lib.ptr(slots), lib.ptr(inv), rows, IH, ID, ratio,
                                   n_keys, max_keys, lib.ptr(qr), lib.ptr(kc), lib.ptr(vis), 0, lib.stream()), "prepare")
    G.gemm_raw(qr, kc, got, rows * IH, n_keys, ID, lda=ID, ldb=ID, ldo=max_keys, out_mode=8, bn=256,
               row_w=w[:, w_off:], row_w_ld=w_stride, col_limit=vis, status=st)
    torch.cuda.synchronize()
    lib.raise_on_status(st, "index gemm")
    for r in (0, 57, rows - 1):
        nv = (pos0 + r + 1) // ratio
        assert int(vis[r]) == nv
        a, b = got[r, :nv], ref[r, :nv]
        assert float((a - b).abs().max()) < 2e-3 * float(b.abs().max())
        assert torch.isinf(got[r, nv:n_keys]).all()


@pytest.mark.parametrize("bn", [32, 64, 128, 256])
@pytest.mark.parametrize("rows,n_keys,static", [(1, 70, 0), (5, 257, 2), (70, 1000, 0), (301, 640, 1)])
def test_index_scores_by_tiles(rows, n_keys, static, bn):
    """Scores whatever the queries of a tile see: nothing, part of a tile, keys beyond the last one; unordered limits."""
    from ds41rt_b200.ops import gemm as G, lib
    IH, ID, ld = 32, 128, 1024
    torch.manual_seed(rows)
    q = torch.randn(rows * IH, ID, device="cuda").bfloat16()
    keys = torch.randn(n_keys, ID, device="cuda").bfloat16()
    w = torch.randn(rows, IH, device="cuda")
    limit = torch.randint(0, n_keys + 20, (rows,), device="cuda", dtype=torch.int32)
    limit[rows // 2:rows // 2 + 9] = 0                     # whole tiles of queries that see nothing
    for lim in (limit, None):
        got = torch.full((rows, ld), float("nan"), device="cuda")
        st = lib.new_status("cuda")
        G.gemm_raw(q, keys, got, rows * IH, n_keys, ID, lda=ID, ldb=ID, ldo=ld, out_mode=8, bn=bn, row_w=w, row_w_ld=IH,
                   col_limit=lim, status=st, static_operand=static)
        torch.cuda.synchronize()
        lib.raise_on_status(st, "index gemm")
        qh = q.double().view(rows, IH, ID)
        want = torch.einsum("rh,rhk->rk", w.double(), (qh @ keys.double().T).relu())
        bound = torch.einsum("rh,rhk->rk", w.double().abs(), qh.abs() @ keys.double().abs().T) * (ID + IH + 2) * 2.0 ** -23
        sees = torch.arange(n_keys, device="cuda")[None] < (lim if lim is not None else limit.new_full((rows,), n_keys))[:, None]
        assert torch.isneginf(got[:, :n_keys][~sees]).all() and got[:, n_keys:].isnan().all()
        assert ((got[:, :n_keys].double() - want).abs() <= bound)[sees].all()


@pytest.mark.parametrize("bn", [32, 64, 128, 256])
def test_index_scores_of_eight_bit_operands(bn):
    """E4M3 queries and keys: products are exact, sums as in the bf16 form."""
    from ds41rt_b200.ops import gemm as G, lib
    IH, ID, rows, n_keys, ld = 32, 128, 37, 300, 512
    torch.manual_seed(bn)
    q = (torch.randn(rows * IH, ID, device="cuda") * 4).to(torch.float8_e4m3fn)
    keys = (torch.randn(n_keys, ID, device="cuda") * 4).to(torch.float8_e4m3fn)
    w, limit = torch.randn(rows, IH, device="cuda"), torch.randint(0, n_keys + 20, (rows,), device="cuda", dtype=torch.int32)
    limit[8:20] = 0
    got, st = torch.full((rows, ld), float("nan"), device="cuda"), lib.new_status("cuda")
    G.gemm_raw(q, keys, got, rows * IH, n_keys, ID, lda=ID, ldb=ID, ldo=ld, kind=1, out_mode=8, bn=bn, row_w=w, row_w_ld=IH,
               col_limit=limit, status=st)
    torch.cuda.synchronize()
    lib.raise_on_status(st, "index gemm")
    qh = q.double().view(rows, IH, ID)
    want = torch.einsum("rh,rhk->rk", w.double(), (qh @ keys.double().T).relu())
    bound = torch.einsum("rh,rhk->rk", w.double().abs(), qh.abs() @ keys.double().abs().T) * (ID + IH + 2) * 2.0 ** -23
    sees = torch.arange(n_keys, device="cuda")[None] < limit[:, None]
    assert torch.isneginf(got[:, :n_keys][~sees]).all() and got[:, n_keys:].isnan().all()
    assert ((got[:, :n_keys].double() - want).abs() <= bound)[sees].all()


def test_fp4_index_keys_and_queries_follow_the_quantisation_oracle():
    """Index keys stored as FP4 rows (E2M1 pairs + UE8M0 per 32 values, 68 bytes for 128 values): the per-key kernel and
    the tensor-core path both score the dequantised keys against queries quantised the same way; the per-key kernel
    also rounds to bf16 where the reference does (dot, weighted relu, head sum)."""
    from ds41rt_b200.config import RopeConfig, rope_inv_freq
    from ds41rt_b200.models.reference import apply_rope
    from ds41rt_b200.ops import gemm as G, lib, quant_ref as Q
    k = lib.kernels()
    torch.manual_seed(9)
    rows, IH, ID, ratio, page_rows, max_pages, max_keys = 70, 32, 128, 2, 32, 40, 1280
    pos0 = 2000
    positions = torch.arange(pos0, pos0 + rows, dtype=torch.int32, device="cuda")
    slots = torch.zeros(rows, dtype=torch.int32, device="cuda")
    ldq = IH * ID
    q = torch.randn(rows, ldq, device="cuda").bfloat16()
    w = torch.rand(rows, IH, device="cuda")
    keys = (torch.randn(max_pages * page_rows, ID, device="cuda") * torch.exp(torch.randn(max_pages * page_rows, 1,
                                                                                             device="cuda"))).bfloat16()
    packed, e = Q.quant_mxfp4(keys.float().cpu(), 32)
    row_bytes = 68
    pool = torch.zeros(max_pages * page_rows, row_bytes, dtype=torch.uint8)
    pool[:, :ID // 2] = packed.view(torch.uint8)
    pool[:, ID // 2:ID // 2 + ID // 32] = e.to(torch.uint8)
    pool = pool.cuda()
    keys_dq = Q.dequant_mxfp4(packed, e, 32).cuda()
    page_table = torch.randperm(max_pages, device="cuda").int().view(1, max_pages).contiguous()
    inv = torch.tensor(rope_inv_freq(RopeConfig(), ID // 2), device="cuda")
    got = torch.full((rows, max_keys), float("nan"), device="cuda")
    lib.check(k.ds41_index_score_cand(lib.ptr(q), C.c_longlong(ldq), 0, lib.ptr(w), IH, 0, lib.ptr(pool),
                                      lib.ptr(page_table), max_pages, page_rows, lib.ptr(positions), lib.ptr(slots),
                                      lib.ptr(inv), rows, IH, ID, ratio, lib.ptr(got), max_keys, None, 0, 0, row_bytes,
                                      lib.stream()), "score")
    n_keys = (pos0 + rows) // ratio
    qr = torch.zeros(rows * IH, ID, device="cuda", dtype=torch.bfloat16)
    kc = torch.zeros(max_keys, ID, device="cuda", dtype=torch.bfloat16)
    vis = torch.zeros(rows, dtype=torch.int32, device="cuda")
    gemm = torch.full((rows, max_keys), float("nan"), device="cuda")
    st = lib.new_status("cuda")
    lib.check(k.ds41_index_prepare(lib.ptr(q), C.c_longlong(ldq), 0, lib.ptr(pool), lib.ptr(page_table), max_pages,
                                   page_rows, lib.ptr(positions), lib.ptr(slots), lib.ptr(inv), rows, IH, ID, ratio,
                                   n_keys, max_keys, lib.ptr(qr), lib.ptr(kc), lib.ptr(vis), row_bytes, lib.stream()),
              "prepare")
    G.gemm_raw(qr, kc, gemm, rows * IH, n_keys, ID, lda=ID, ldb=ID, ldo=max_keys, out_mode=8, bn=256, row_w=w,
               row_w_ld=IH, col_limit=vis, status=st)
    torch.cuda.synchronize()
    lib.raise_on_status(st, "index gemm")
    # oracle: RoPE, bf16, FP4 round trip of the queries; keys as dequantised; logical key c lives in page_table[c / page_rows]
    qh = q.float().view(rows, IH, ID).cpu()
    qh = apply_rope(qh, positions.cpu().long(), inv.cpu(), ID // 2).bfloat16().float()
    qh = Q.qdq_mxfp4(qh, 32).cuda()
    logical = torch.arange(n_keys, device="cuda")
    phys = page_table[0, logical // page_rows].long() * page_rows + logical % page_rows
    kd = keys_dq[phys]
    assert torch.equal(kc[:n_keys].float(), kd)                                  # gathered keys are the dequantised rows
    # the queries are FP4 values (a fixed point of the round trip) and the round trip of the oracle's RoPE'd queries, up to
    # the few elements where the kernel's and torch's sine differ by an ulp of bf16 before quantisation
    qk = qr.float().view(rows, IH, ID)
    assert torch.equal(Q.qdq_mxfp4(qk.cpu(), 32).cuda(), qk)
    assert float((qk == qh).float().mean()) > 0.97 and float((qk - qh).abs().max()) <= 0.5 * float(qh.abs().max())
    qh = qk
    bf = lambda t: t.bfloat16().float()
    dots = bf(torch.einsum("rhd,cd->rhc", qh, kd))
    want = bf((bf(torch.relu(dots) * w[:, :, None])).sum(1))
    for r in (0, 33, rows - 1):
        nv = (pos0 + r + 1) // ratio
        a, b = got[r, :nv], want[r, :nv]
        assert float((a - b).abs().max()) <= 0.02 * float(b.abs().max())        # bf16 rounding points: one ulp apart at most
        g = gemm[r, :nv]
        assert float((g - b).abs().max()) < 0.02 * float(b.abs().max())
        assert torch.isinf(gemm[r, nv:n_keys]).all()


def test_nvfp4_activation_quantiser_matches_oracle():
    from ds41rt_b200.ops import lib, quant_ref as Q
    from ds41rt_b200.ops.mx import pack_sf_atoms
    k = lib.kernels()
    torch.manual_seed(5)
    rows, K = 70, 768
    x = (torch.randn(rows, K, device="cuda") * torch.exp(torch.randn(rows, 1, device="cuda"))).bfloat16()
    gs = float(x.float().abs().amax() / (448 * 6))
    want_q, want_s, _ = Q.quant_nvfp4(x.float(), gs)
    q = torch.zeros(rows, K // 2, dtype=torch.uint8, device="cuda")
    sf = torch.zeros((rows + 127) // 128, K // 64, 512, dtype=torch.uint8, device="cuda")
    lib.check(k.ds41_act_quant_nvfp4_rows(lib.ptr(x), C.c_longlong(K), lib.ptr(q), C.c_longlong(K), lib.ptr(sf), rows,
                                          K, C.c_float(gs), None, 1, C.c_longlong(0), C.c_longlong(0), C.c_longlong(0), None,
                                          lib.stream()), "quant")
    torch.cuda.synchronize()
    assert torch.equal(q, want_q)
    want_atoms = pack_sf_atoms(want_s.view(torch.uint8))
    from ds41rt_b200.ops.mx import unpack_sf_atoms
    assert torch.equal(unpack_sf_atoms(sf.cpu(), rows), unpack_sf_atoms(want_atoms.cpu(), rows))


def test_candidate_blocks_select_and_restrict():
    """Candidate layer: block maxima, newest block pinned, best blocks kept (ties to the lowest block id) -> list + mask;
    the masked top-k then only sees keys of those blocks."""
    from ds41rt_b200.ops import lib
    k = lib.kernels()
    rows, max_keys, B, KB, topk = 5, 3000, 8, 40, 64
    torch.manual_seed(1)
    scores = torch.randn(rows, max_keys, device="cuda")
    scores[1] = scores[1].round()                                  # ties between block maxima
    pos = torch.tensor([2999, 2500, 100, 1203, 9], dtype=torch.int32, device="cuda")   # row 2: fewer blocks than KB
    slot = torch.tensor([0, 0, 0, 0, -1], dtype=torch.int32, device="cuda")
    nb = (max_keys + B - 1) // B
    words = (nb + 31) // 32
    blocks = torch.zeros(rows, KB, dtype=torch.int32, device="cuda")
    n_blocks = torch.zeros(rows, dtype=torch.int32, device="cuda")
    mask = torch.full((rows, words), -1, dtype=torch.int32, device="cuda")
    lib.check(k.ds41_candidate_select(lib.ptr(scores), max_keys, lib.ptr(pos), lib.ptr(slot), 1, B, KB, lib.ptr(blocks),
                                      lib.ptr(n_blocks), lib.ptr(mask), words, rows, lib.stream()), "candidate_select")
    sel = torch.zeros(rows, topk, dtype=torch.int32, device="cuda")
    n_sel = torch.zeros(rows, dtype=torch.int32, device="cuda")
    scores2 = torch.randn(rows, max_keys, device="cuda")           # a later layer's scores
    lib.check(k.ds41_topk_select_cand(lib.ptr(scores2), max_keys, lib.ptr(pos), lib.ptr(slot), 1, topk, lib.ptr(sel),
                                      lib.ptr(n_sel), rows, lib.ptr(mask), words, B, lib.stream()), "topk_cand")
    torch.cuda.synchronize()
    bits = mask.cpu().numpy().view("uint32")
    for r in range(4):
        n = int(pos[r]) + 1
        nbv = (n + B - 1) // B
        s = scores[r, :n].cpu()
        s = torch.nn.functional.pad(s, (0, nbv * B - n), value=float("-inf")).view(nbv, B).amax(-1)
        s[(n - 1) // B] = float("inf")
        want = sorted(torch.sort(s, descending=True, stable=True).indices[:KB].tolist())
        got = blocks[r, : int(n_blocks[r])].tolist()
        assert got == want, r
        on = [b for b in range(nb) if (int(bits[r, b >> 5]) >> (b & 31)) & 1]
        assert on == want
        # restricted selection of the later layer
        allowed = torch.zeros(n, dtype=torch.bool)
        for b in want:
            allowed[b * B: (b + 1) * B] = True
        s2 = scores2[r, :n].cpu().masked_fill(~allowed, float("-inf"))
        n_ok = int(allowed.sum())
        order = torch.sort(s2, descending=True, stable=True).indices[: min(topk, n_ok)]
        assert sel[r, : int(n_sel[r])].tolist() == sorted(order.tolist()), r
        assert int(n_sel[r]) == min(topk, n_ok)
    assert int(n_blocks[4]) == 0 and int(n_sel[4]) == 0 and not bits[4].any()


@pytest.mark.parametrize("rows,H", [(300, 512), (1024, 1024)])
def test_hc_mixes_on_the_tensor_cores_match_the_dot_product_kernel(rows, H):
    """Long-pass form of the hyper-connection step: expand without the mixing matrix, the 24 projections from a
    tcgen05 GEMM over the stored streams with the matrix as bf16 high + low parts, hc_finish reading the split-K
    planes.  Streams are identical to the dot-product kernel's; pre / post / comb and the normalised rows agree to
    fp32 rounding of a 4H-long sum, and with the fp32 oracle as closely as the dot-product kernel does."""
    from ds41rt_b200.models import reference as R
    from ds41rt_b200.ops import gemm as G
    from ds41rt_b200.ops import lib
    k = lib.kernels()
    torch.manual_seed(rows)
    K = 4 * H
    streams = torch.randn(rows, 4, H, device="cuda").bfloat16()
    sub = torch.randn(2, rows, H, device="cuda")
    fn = torch.randn(24, K, device="cuda") * 0.5
    scale = torch.tensor([1.0, 0.7, 1.3], device="cuda")
    base = torch.randn(24, device="cuda") * 0.5
    pre_in = torch.rand(rows, 4, device="cuda")
    norm_w = torch.rand(H, device="cuda") + 0.5
    post = torch.rand(rows, 4, device="cuda") * 2
    comb = torch.rand(rows, 16, device="cuda") / 4
    st = lib.new_status("cuda")
    bases = (C.c_void_p * 1)(sub.data_ptr())

    def run(tc, fused=False):
        s = streams.clone()
        partial = torch.zeros(H // 128, rows, 25, device="cuda")
        outs = [torch.zeros(rows, 4, device="cuda"), torch.zeros(rows, 4, device="cuda"),
                torch.zeros(rows, 16, device="cuda"), torch.zeros(rows, H, device="cuda", dtype=torch.bfloat16)]
        tap = torch.zeros(rows, H, device="cuda")
        collapse = (lib.ptr(pre_in), lib.ptr(norm_w), lib.ptr(outs[3]), lib.ptr(tap), C.c_float(1e-20)) if fused else \
            (lib.ptr(None), lib.ptr(None), lib.ptr(None), lib.ptr(None), C.c_float(0.0))
        lib.check(k.ds41_hc_post_mix(lib.ptr(s), lib.ptr(s), bases, 1, 2, C.c_longlong(rows * H), lib.ptr(post),
                                     lib.ptr(comb), lib.ptr(None if tc else fn), lib.ptr(partial), rows, H,
                                     lib.ptr(None), lib.ptr(None), lib.ptr(st), *collapse, lib.stream()), "post_mix")
        mix = (lib.ptr(None), 0, C.c_longlong(0), 0)
        keep = None
        if tc:
            hi = fn.bfloat16()
            w = torch.zeros(64, K, device="cuda", dtype=torch.bfloat16)
            w[:24], w[24:48] = hi, (fn - hi.float()).bfloat16()
            splits = G.pick_splits(rows, K, max_splits=16)
            assert splits > 1
            planes = torch.zeros(splits, rows, 64, device="cuda")
            G.gemm_raw(s.view(rows, K), w, None, rows, 64, K, lda=K, ldb=K, ldo=64, out_mode=1, k_splits=splits,
                       split_workspace=planes, bn=64, status=st, static_operand=2)
            mix = (lib.ptr(planes), splits, C.c_longlong(rows * 64), 64)
            keep = (w, planes)
        lib.check(k.ds41_hc_finish(lib.ptr(partial), 1 if tc else H // 128, lib.ptr(scale), lib.ptr(base), lib.ptr(pre_in),
                                   lib.ptr(s), lib.ptr(norm_w), lib.ptr(outs[0]), lib.ptr(outs[1]), lib.ptr(outs[2]),
                                   lib.ptr(None if fused else outs[3]), lib.ptr(None if fused else tap), lib.ptr(None),
                                   lib.ptr(None), rows, H, 20, C.c_float(1e-6), C.c_float(1e-20), *mix, lib.stream()),
                  "finish")
        torch.cuda.synchronize()
        lib.raise_on_status(st, "hc mixes")
        return s, outs + [tap], partial, keep

    s_a, a, part_a, _ = run(False)
    s_b, b, part_b, _ = run(True)
    s_c, c, part_c, _ = run(True, fused=True)       # expand kernel also collapses and normalises; finish: mixes only
    assert torch.equal(s_a, s_b) and torch.equal(s_b, s_c)
    assert torch.equal(b[3], c[3]) and torch.equal(b[4], c[4]) and torch.equal(part_b[0, :, 24], part_c[0, :, 24])
    for x, y in zip(b[:3], c[:3]):
        assert float((x - y).abs().max()) < 1e-5          # the split-K planes are summed in another order
    assert torch.allclose(part_a[:, :, 24].sum(0), part_b[0, :, 24], rtol=1e-5, atol=1e-4)   # sums of squares
    assert torch.equal(a[3], b[3])                                                       # collapse + norm: same inputs
    for x, y in zip(a[:3], b[:3]):
        assert float((x - y).abs().max()) < 2e-4
    pre1, post1, comb1 = R.hc_mixes(s_b.float().cpu(), fn.cpu(), scale.cpu(), base.cpu(), 4, 20, 1e-6, 1e-20)
    assert float((b[0].cpu() - pre1).abs().max()) < 1e-3
    assert float((b[1].cpu() - post1).abs().max()) < 1e-3
    assert float((b[2].cpu().view(rows, 4, 4) - comb1).abs().max()) < 1e-3


@pytest.mark.parametrize("kind,K", [("mx", 128), ("mx", 640), ("mx", 2304), ("nvfp4", 64), ("nvfp4", 768), ("nvfp4", 5120)])
def test_tile_quantisers_touch_the_rows_of_the_table(kind, K):
    """Groups on 128-row boundaries with ragged tails: the table's rows are those of the host oracle, bit for bit, and every
    other byte stays as it was."""
    from ds41rt_b200.ops import lib, quant_ref as Q
    from ds41rt_b200.ops.mx import pack_sf_atoms, unpack_sf_atoms
    k = lib.kernels()
    torch.manual_seed(K)
    sizes, bn = [1, 128, 0, 127, 9, 65], 64
    rows, row0, end = 0, [], []
    for n in sizes:
        for r in range(rows, rows + n, bn):
            row0.append(r)
            end.append(min(r + bn, rows + n))
        rows += (n + 127) // 128 * 128
    live = torch.cat([torch.arange(a, b) for a, b in zip(row0, end)])
    i32 = dict(dtype=torch.int32, device="cuda")
    t0, t1, n = torch.tensor(row0 + [0] * 4, **i32), torch.tensor(end + [rows] * 4, **i32), torch.tensor([len(row0)], **i32)
    x = (torch.randn(rows, K, device="cuda") * torch.exp(torch.randn(rows, 1, device="cuda"))).bfloat16()
    table = lib.ptr(t0), lib.ptr(t1), lib.ptr(n), len(row0) + 4, lib.stream()
    per = 128 if kind == "mx" else 64                      # columns of a scale atom
    q = torch.full((rows, K if kind == "mx" else K // 2), 0xAB, dtype=torch.uint8, device="cuda")
    sf = torch.full((rows // 128, K // per, 512), 0xAB, dtype=torch.uint8, device="cuda")
    head = lib.ptr(x), C.c_longlong(K), lib.ptr(q), C.c_longlong(K), lib.ptr(sf), rows, K
    if kind == "mx":
        lib.check(k.ds41_act_quant_mx_tiles(*head, *table), "quant")
        want = torch.zeros(rows, K, dtype=torch.uint8, device="cuda")
        want_sf = torch.zeros_like(sf)
        lib.check(k.ds41_act_quant_mx(lib.ptr(x), C.c_longlong(K), C.c_longlong(0), lib.ptr(want), C.c_longlong(K),
                                      C.c_longlong(0), lib.ptr(want_sf), C.c_longlong(0), rows, K, 1, 128, None, lib.stream()),
                  "quant")
    else:
        gs = float(x.float().abs().amax() / (448 * 6))
        lib.check(k.ds41_act_quant_nvfp4_tiles(*head, C.c_float(gs), *table), "quant")
        want, want_s, _ = Q.quant_nvfp4(x.float(), gs)
        want_sf = pack_sf_atoms(want_s.view(torch.uint8))
    torch.cuda.synchronize()
    dead = torch.ones(rows, dtype=torch.bool)
    dead[live] = False
    got_s, want_s = unpack_sf_atoms(sf.cpu(), rows), unpack_sf_atoms(want_sf.cpu(), rows)
    assert torch.equal(q.cpu()[live], want.cpu()[live]) and bool((q.cpu()[dead] == 0xAB).all())
    assert torch.equal(got_s[live], want_s[live]) and bool((got_s[dead] == 0xAB).all())


@pytest.mark.parametrize("rows,live,K,pad", [(1, None, 128, 0), (9, 5, 640, 8), (300, None, 384, 0), (1500, 1291, 256, 16)])
def test_row_quantiser_of_long_passes(rows, live, K, pad):
    """Rows below the device count as the general quantiser gives them, bit for bit; what lies behind stays as it was."""
    from ds41rt_b200.ops import lib
    from ds41rt_b200.ops.mx import unpack_sf_atoms
    k = lib.kernels()
    torch.manual_seed(rows)
    x = (torch.randn(rows, K + pad, device="cuda") * torch.exp(torch.randn(rows, 1, device="cuda"))).bfloat16()
    q, want = (torch.full((rows, K), 0xAB, dtype=torch.uint8, device="cuda") for _ in range(2))
    sf, want_sf = (torch.full(((rows + 127) // 128, K // 128, 512), 0xAB, dtype=torch.uint8, device="cuda") for _ in range(2))
    n = None if live is None else torch.tensor([live], dtype=torch.int32, device="cuda")
    lib.check(k.ds41_act_quant_mx_rows(lib.ptr(x), C.c_longlong(K + pad), lib.ptr(q), C.c_longlong(K), lib.ptr(sf), rows, K,
                                       lib.ptr(n), lib.stream()), "quant")
    m = rows if live is None else live
    lib.check(k.ds41_act_quant_mx(lib.ptr(x), C.c_longlong(K + pad), C.c_longlong(0), lib.ptr(want), C.c_longlong(K),
                                  C.c_longlong(0), lib.ptr(want_sf), C.c_longlong(0), m, K, 1, 128, None, lib.stream()), "quant")
    torch.cuda.synchronize()
    assert torch.equal(q, want)
    a, b = unpack_sf_atoms(sf.cpu(), rows), unpack_sf_atoms(want_sf.cpu(), rows)
    assert torch.equal(a[:m], b[:m]) and bool((a[m:] == 0xAB).all())


@pytest.mark.parametrize("vocab,ld,rows", [(3, 3, 1), (31, 32, 2), (4096, 4096, 3), (65537, 65540, 2), (129280, 129280, 5)])
def test_argmax_rows_over_a_cluster(vocab, ld, rows):
    """Largest allowed logit, lowest id among equals, at the edges of the eight parts of a row; statuses."""
    from ds41rt_b200.ops import lib
    k = lib.kernels()
    torch.manual_seed(vocab)
    logits = torch.randn(rows, ld, device="cuda")
    per = -(-(-(-vocab // 8)) // 4) * 4
    for i, at in enumerate((vocab - 1, 0, min(per, vocab - 1), min(2 * per - 1, vocab - 1), vocab // 2)[:rows]):
        logits[i, at] = 50.0
        logits[i, min(at + per, vocab - 1)] = 50.0                  # the same value in a later part
    words = (vocab + 31) // 32
    mask = torch.full((rows, words), -1, dtype=torch.int32, device="cuda")
    if rows > 1:
        mask[1] = 0
    best, idx = torch.zeros(rows, device="cuda"), torch.zeros(rows, dtype=torch.int32, device="cuda")
    status = torch.full((rows,), -1, dtype=torch.int32, device="cuda")
    for m in (None, mask):
        lib.check(k.ds41_argmax_rows(lib.ptr(logits), C.c_longlong(ld), rows, vocab, 0, lib.ptr(m), words, lib.ptr(best),
                                     lib.ptr(idx), lib.ptr(status), lib.stream()), "argmax")
        torch.cuda.synchronize()
        want = logits[:, :vocab].cpu()
        for r in range(rows):
            if m is not None and r == 1:
                assert int(idx[r]) == -1 and int(status[r]) == 2
            else:
                top = want[r].max()
                assert int(idx[r]) == int((want[r] == top).nonzero()[0]) and float(best[r]) == float(top) and int(status[r]) == 0
    logits[rows - 1, vocab - 1] = float("nan")
    lib.check(k.ds41_argmax_rows(lib.ptr(logits), C.c_longlong(ld), rows, vocab, 0, None, words, lib.ptr(best), lib.ptr(idx),
                                 lib.ptr(status), lib.stream()), "argmax")
    torch.cuda.synchronize()
    assert status.tolist() == [0] * (rows - 1) + [1]


@pytest.mark.parametrize("rows,splits,E,I_sh", [(512, 3, 384, 64), (513, 1, 36, 4), (777, 1, 512, 0), (2049, 1, 384, 2304)])
def test_router_rows(rows, splits, E, I_sh):
    """A warp per row: experts, order (ties to the lowest id, masked experts last) and weights of the plain statement."""
    from ds41rt_b200.ops import lib
    from ds41rt_b200.models import reference as R
    k = lib.kernels()
    torch.manual_seed(rows)
    topk = 6
    planes = torch.randn(splits, rows, E + 2 * I_sh, device="cuda")
    planes[:, 1, :E] = 0.25                                          # every score alike
    bias = torch.zeros(E, device="cuda")
    bias[E // 2:] = float("-inf")
    ids = torch.full((rows, topk), -7, dtype=torch.int32, device="cuda")
    wts = torch.zeros(rows, topk, device="cuda")
    act = torch.zeros(rows, max(I_sh, 1), device="cuda", dtype=torch.bfloat16)
    lib.check(k.ds41_router_select(lib.ptr(planes), splits, rows, E + 2 * I_sh, E, I_sh, topk, lib.ptr(bias), C.c_float(1.5),
                                   C.c_float(10.0), lib.ptr(ids), lib.ptr(wts), lib.ptr(act), lib.stream()), "router")
    torch.cuda.synchronize()
    total = planes[0].clone()
    for s in range(1, splits):
        total += planes[s]
    total = total.cpu()
    score = torch.sqrt(torch.nn.functional.softplus(total[:, :E]))
    order = torch.sort(score + bias.cpu(), dim=-1, descending=True, stable=True)
    gap = (order.values[:, :topk] - order.values[:, 1:topk + 1]).min(-1).values
    clear = gap > 1e-5                                               # log1p / sqrt differ in the last places
    clear[1] = True
    assert int(clear.sum()) > rows * 0.9
    want = order.indices[:, :topk]
    assert torch.equal(ids.cpu().long()[clear], want[clear])
    sel = torch.gather(score, 1, want)
    assert ((wts.cpu() - sel / sel.sum(-1, keepdim=True) * 1.5)[clear]).abs().max() < 1e-5
    if I_sh:
        w = R.swiglu_clamped(total[:, E:E + I_sh].bfloat16().float(), total[:, E + I_sh:].bfloat16().float(), 10.0)
        # one rounding to bf16 (2^-9) and the fast exponential's few units of 2^-23
        assert ((act.float().cpu() - w).abs() <= w.abs() * 2.0 ** -8 + 1e-6).all()


@pytest.mark.parametrize("tokens,width", [(400, 128), (500, 192), (690, 192), (760, 128), (1160, 192)])
def test_expert_tile_width_by_pass_size(tokens, width):
    """Passes that take 192-token tiles (second tiles in mid-atom, the last expert's at the buffer's end) and passes that take
    128-token ones give the rows of a layer whose tiles are 128 tokens wide, bit for bit."""
    from ds41rt_b200.models.ds41 import quantize_expert_stack
    from ds41rt_b200.parallel.ep import ExpertParallelMoE
    from ds41rt_b200.parallel.fabric import Fabric
    torch.manual_seed(tokens)
    E, H, I, topk = 8, 1792, 2432, 2                     # large enough for wide tiles
    dev = torch.device("cuda", 0)
    w13, sf13 = quantize_expert_stack(torch.randn(E, 2 * I, H) * 0.05, dev)
    w2, sf2 = quantize_expert_stack(torch.randn(E, H, I) * 0.05, dev)
    x = torch.randn(tokens, H, device=dev).bfloat16()
    p = torch.rand(tokens, E, device=dev)
    p[:, E - 1] += 0.3                                   # the last expert holds more than its share
    ids = p.topk(topk, -1).indices.int().contiguous()
    wts = torch.rand(tokens, topk, device=dev)
    got = []
    for tile in (None, 128):
        ep = ExpertParallelMoE(Fabric.single(dev), w13, w2, topk=topk, max_tokens=tokens, w13_sf=sf13, w2_sf=sf2, tile_tokens=tile)
        out = torch.zeros(tokens, H, device=dev)
        ep.forward(x, ids, wts, out)
        torch.cuda.synchronize()
        ep.check()
        assert ep.bn == (width if tile is None else 128)
        got.append(out)
    assert torch.equal(got[0], got[1]) and float(got[0].abs().max()) > 0


@pytest.mark.parametrize("H,rows,expand,tap", [(128, 256, True, True), (5120, 300, True, False), (5120, 1000, False, False),
                                               (6144, 450, True, True)])
def test_expand_of_long_passes_matches_short_ones(H, rows, expand, tap):
    """Rows through the ring of bulk copies (in place, uneven rows per CTA) are the rows of a block each, bit for bit."""
    from ds41rt_b200.ops import lib
    k = lib.kernels()
    torch.manual_seed(H + rows)
    start = torch.randn(rows, 4, H, device="cuda").bfloat16()
    plane, post, comb = torch.randn(rows, H, device="cuda"), torch.rand(rows, 4, device="cuda"), torch.rand(rows, 16, device="cuda")
    pre, norm_w, st = torch.rand(rows, 4, device="cuda"), torch.rand(H, device="cuda"), lib.new_status(torch.device("cuda", 0))
    got = []
    for most in (rows, 150):                               # one pass; passes that are too small for the ring
        s, xn = start.clone(), torch.zeros(rows, H, device="cuda", dtype=torch.bfloat16)
        partial, mean = torch.zeros(rows, 25, device="cuda"), torch.zeros(rows, H, device="cuda")
        for r0 in range(0, rows, most):
            n = min(most, rows - r0)
            bases = (C.c_void_p * 1)(plane[r0:].data_ptr())
            lib.check(k.ds41_hc_post_mix(lib.ptr(s[r0:]), lib.ptr(s[r0:]), bases, int(expand), 1, C.c_longlong(0),
                                         lib.ptr(post[r0:]), lib.ptr(comb[r0:]), lib.ptr(None), lib.ptr(partial[r0:]), n, H,
                                         lib.ptr(None), lib.ptr(None), lib.ptr(st), lib.ptr(pre[r0:]), lib.ptr(norm_w),
                                         lib.ptr(xn[r0:]), lib.ptr(mean[r0:] if tap else None), C.c_float(1e-6), lib.stream()), "expand")
        torch.cuda.synchronize()
        assert int(st[0]) == 0
        got.append((s, xn, partial, mean))
    for a, b in zip(*got):
        assert torch.equal(a, b)
    assert float(got[0][1].float().abs().max()) > 0 and torch.equal(got[0][0], start) == (not expand)


@pytest.mark.parametrize("vocab,ld,rows", [(16383, 16384, 5), (16384, 16384, 16), (16384, 16384, 17), (4096, 4096, 3), (131072, 131072, 128),
                                           (131072, 131072, 129)])
def test_argmax_rows_on_both_sides_of_the_rule(vocab, ld, rows):
    """A cluster for few long rows, one block for short or many ones."""
    test_argmax_rows_over_a_cluster(vocab, ld, rows)


@pytest.mark.parametrize("rows,splits,E,I_sh", [(512, 3, 384, 64), (512, 4, 384, 64), (640, 4, 36, 4), (1919, 12, 64, 0), (1920, 12, 64, 0)])
def test_router_rows_do_not_depend_on_the_pass(rows, splits, E, I_sh):
    """A long pass, by warps or (with many planes) by blocks, gives every row what a short pass gives it, bit for bit."""
    from ds41rt_b200.ops import lib
    k = lib.kernels()
    torch.manual_seed(rows)
    topk, ntot = 6, E + 2 * I_sh
    planes, bias = torch.randn(splits, rows, ntot, device="cuda"), torch.randn(E, device="cuda") * 0.1
    planes[:, 3, :E] = 0.5
    planes[0, 5, 0] = float("inf")

    def run(part):
        n = part.shape[1]
        part = part.contiguous()
        ids, wts = torch.zeros(n, topk, dtype=torch.int32, device="cuda"), torch.zeros(n, topk, device="cuda")
        act = torch.zeros(n, max(I_sh, 1), device="cuda", dtype=torch.bfloat16)
        lib.check(k.ds41_router_select(lib.ptr(part), splits, n, ntot, E, I_sh, topk, lib.ptr(bias), C.c_float(1.5), C.c_float(10.0),
                                       lib.ptr(ids), lib.ptr(wts), lib.ptr(act), lib.stream()), "router")
        torch.cuda.synchronize()
        return ids, wts.view(torch.int32), act.view(torch.int16)

    whole, parts = run(planes), [run(planes[:, r:r + 100]) for r in range(0, rows, 100)]
    for i, w in enumerate(whole):
        assert torch.equal(w, torch.cat([p[i] for p in parts]))


@pytest.mark.parametrize("rows", [296, 297])
@pytest.mark.parametrize("expand", [False, True])
def test_expand_on_both_sides_of_the_rule(rows, expand):
    """Two blocks an SM still hold 296 rows at once on 148 SMs; one more goes through the ring."""
    test_expand_of_long_passes_matches_short_ones(1024, rows, expand, True)


@pytest.mark.parametrize("rows,H,splits", [(55, 1024, 1), (56, 1024, 16), (11, 5120, 4), (12, 5120, 4), (3, 6272, 2), (9, 6272, 2),
                                           (7, 7168, 1), (8, 7168, 16)])
def test_hc_step_rows_do_not_depend_on_the_pass(rows, H, splits):
    """Small grids hold their operands in registers, larger ones load them when needed; rows beyond 6144 columns go on in
    further pieces.  Every row is what a launch of its own gives, bit for bit, and what the plain statement gives."""
    from ds41rt_b200.models import reference as R
    from ds41rt_b200.ops import lib
    k = lib.kernels()
    torch.manual_seed(rows + H)
    streams, sub = torch.randn(rows, 4, H, device="cuda").bfloat16(), torch.randn(splits, rows, H, device="cuda")
    fn, scale, base = torch.randn(24, 4 * H, device="cuda") * 0.02, torch.tensor([1.0, 0.7, 1.3], device="cuda"), torch.randn(24, device="cuda") * 0.5
    pre, post = torch.rand(rows, 4, device="cuda"), torch.rand(rows, 4, device="cuda") * 2
    comb, norm_w = torch.rand(rows, 16, device="cuda") * 0.5, torch.rand(H, device="cuda") + 0.5
    st = lib.new_status("cuda")

    def run(r0, r1):
        n = r1 - r0
        part = sub[:, r0:r1].contiguous()
        bases = (C.c_void_p * 1)(part.data_ptr())
        src, p_in, p_out, cb = (t[r0:r1].contiguous() for t in (streams, pre, post, comb))
        z = lambda *s, dt=torch.float32: torch.zeros(*s, device="cuda", dtype=dt)
        out = [torch.empty_like(src), z(n, 4), z(n, 4), z(n, 16), z(n, H, dt=torch.bfloat16), z(n, H, dt=torch.uint8), z(n, H)]
        scratch = [z(H // 128, n, 26), z(n, H), z(n, dt=torch.int32), z(1, H // 128, 512, dt=torch.uint8)]
        a = lib.HcStepArgs()
        a.streams_in, a.part_bases = lib.ptr(src), C.cast(bases, C.c_void_p)
        a.streams_out, a.next_pre, a.post_out, a.comb_out, a.xn, a.xq, a.tap_mean = (lib.ptr(t) for t in out)
        a.partial, a.xc, a.tickets, a.xq_sf = (lib.ptr(t) for t in scratch)
        a.post, a.comb, a.pre_in, a.fn, a.scale, a.base, a.norm_w = (lib.ptr(t) for t in (p_out, cb, p_in, fn, scale, base, norm_w))
        a.status, a.split_stride, a.n_ranks, a.n_splits = lib.ptr(st), n * H, 1, splits
        a.rows, a.H, a.iters, a.hc_eps, a.norm_eps = n, H, 20, 1e-6, 1e-20
        lib.check(k.ds41_hc_step(C.byref(a), lib.stream()), "hc_step")
        torch.cuda.synchronize()
        assert not bool(scratch[2].any())
        return out

    whole, single = run(0, rows), [run(r, r + 1) for r in range(rows)]
    for i, w in enumerate(whole):
        assert torch.equal(w, torch.cat([s[i] for s in single])), i
    y = sub.sum(0).bfloat16().double()
    new = torch.einsum("rsd,rsh->rdh", comb.view(rows, 4, 4).double(), streams.double()) + post.double()[..., None] * y[:, None]
    x = torch.einsum("rs,rsh->rh", pre.double(), whole[0].double())
    xn = x * torch.rsqrt((x * x).mean(-1, keepdim=True)) * norm_w.double()
    assert float((whole[0].double() - new).abs().max()) < 2.0 ** -7 * float(new.abs().max())
    assert float((whole[4].double() - xn).abs().max()) < 2.0 ** -6 * float(xn.abs().max())


def test_qkv_post_refuses_rows_at_odd_columns():
    """kv columns are read in pairs: an odd row length with further rows or planes, or a base between pairs, is refused."""
    from ds41rt_b200.ops import lib
    k = lib.kernels()
    Q, D = 64, 64

    def call(splits, rows, ntot, offset=0):
        planes, one = torch.zeros(splits * rows * ntot + 4, device="cuda"), torch.ones(256, device="cuda")
        i32 = torch.zeros(4, dtype=torch.int32, device="cuda")
        out = torch.zeros(4, 2048, device="cuda")
        err = k.ds41_qkv_post(C.c_void_p(planes.data_ptr() + offset), splits, rows, ntot, Q, D, 32, 0, 0, C.c_float(1.0), lib.ptr(one),
                              lib.ptr(one), lib.ptr(one), lib.ptr(i32), lib.ptr(i32), lib.ptr(out[0]), lib.ptr(out[1]), 4,
                              lib.ptr(out[2]), C.c_float(1e-6), 0, lib.stream())
        torch.cuda.synchronize()
        return err

    assert call(1, 2, 129) != 0 and call(2, 1, 129) != 0 and call(1, 1, 128, offset=4) != 0
    assert call(1, 1, 129) == 0 and call(2, 3, 130) == 0


@pytest.mark.parametrize("rows,Q,extra", [(1, 1280, 0), (3, 2048, 6), (2, 96, 256), (2, 1280, 258), (2, 300, 1300)])
def test_qkv_post_sums_planes_in_their_order(rows, Q, extra):
    """Few planes (columns inside) and many (planes inside), extras in the kv block and in one of their own: the same bits, since
    further planes of zeros change no sum."""
    from ds41rt_b200.ops import lib
    k = lib.kernels()
    torch.manual_seed(Q + extra)
    D, rope, heads = 512, 64, min(extra, 4)
    ntot = Q + D + extra
    planes = torch.randn(5, rows, ntot, device="cuda")
    qn, kn, inv = torch.rand(Q, device="cuda") + 0.5, torch.rand(D, device="cuda") + 0.5, torch.rand(rope // 2, device="cuda")
    pos, slot = torch.arange(7, 7 + rows, dtype=torch.int32, device="cuda"), torch.zeros(rows, dtype=torch.int32, device="cuda")
    got = []
    for n in (5, 7, 8, 16):
        pl = torch.zeros(n, rows, ntot, device="cuda")
        pl[:5] = planes
        ql, win = torch.zeros(rows, Q, device="cuda", dtype=torch.bfloat16), torch.zeros(1, 32, D, device="cuda", dtype=torch.bfloat16)
        ex = torch.full((rows, extra + 1), 7.0, device="cuda")
        lib.check(k.ds41_qkv_post(lib.ptr(pl), n, rows, ntot, Q, D, rope, extra, heads, C.c_float(0.25), lib.ptr(qn), lib.ptr(kn),
                                  lib.ptr(inv), lib.ptr(pos), lib.ptr(slot), lib.ptr(ql), lib.ptr(win), 32, lib.ptr(ex),
                                  C.c_float(1e-6), 0, lib.stream()), "qkv_post")
        torch.cuda.synchronize()
        got.append((ql, win, ex))
    for g in got[1:]:
        assert all(torch.equal(a, b) for a, b in zip(got[0], g))
    total = planes[0].clone()
    for p in planes[1:]:
        total += p
    want = total[:, Q + D:].clone()
    want[:, extra - heads:] *= 0.25
    ql, win, ex = got[0]
    assert torch.equal(ex.view(-1)[: rows * extra].view(rows, extra), want) and bool((ex.view(-1)[rows * extra:] == 7.0).all())
    q = total[:, :Q].bfloat16().double()
    ref = q * torch.rsqrt((q * q).mean(-1, keepdim=True) + 1e-6) * qn.double()
    assert float((ql.double() - ref).abs().max()) < 2.0 ** -7 * float(ref.abs().max())
    assert bool(win[0, 7:7 + rows].any(-1).all()) and not bool(win[0, :7].any())


@pytest.mark.parametrize("splits", [1, 2, 3, 5, 9])
@pytest.mark.parametrize("rows", [222, 223, 600])
@pytest.mark.parametrize("Q,extra", [(1280, 0), (192, 258), (2048, 32)])
def test_qkv_post_of_many_rows(rows, splits, Q, extra):
    """The rows of a long pass hold the bits that each of them gets in a pass of few."""
    from ds41rt_b200.ops import lib
    k = lib.kernels()
    torch.manual_seed(rows + splits)
    D, rope, ring = 512, 64, 640
    ntot = Q + D + extra
    planes = torch.randn(splits, rows, ntot, device="cuda")
    qn, kn, inv = torch.rand(Q, device="cuda") + 0.5, torch.rand(D, device="cuda") + 0.5, torch.rand(rope // 2, device="cuda")
    pos, slot = torch.arange(rows, dtype=torch.int32, device="cuda"), torch.zeros(rows, dtype=torch.int32, device="cuda")
    got = []
    for step in (rows, 75):
        ql, win = torch.zeros(rows, Q, device="cuda", dtype=torch.bfloat16), torch.zeros(1, ring, D, device="cuda", dtype=torch.bfloat16)
        ex = torch.zeros(rows, max(extra, 1), device="cuda")
        for r in range(0, rows, step):
            n = min(step, rows - r)
            part = planes[:, r:r + n].contiguous()
            lib.check(k.ds41_qkv_post(lib.ptr(part), splits, n, ntot, Q, D, rope, extra, min(extra, 4), C.c_float(0.25), lib.ptr(qn),
                                      lib.ptr(kn), lib.ptr(inv), lib.ptr(pos[r:]), lib.ptr(slot[r:]), lib.ptr(ql[r:]), lib.ptr(win),
                                      ring, lib.ptr(ex[r:]), C.c_float(1e-6), 0, lib.stream()), "qkv_post")
        torch.cuda.synchronize()
        got.append((ql, win, ex))
    assert bool(got[0][0].any(1).all()) and bool(got[0][1][0, :rows].any(1).all())
    assert all(torch.equal(a, b) for a, b in zip(*got))


@pytest.mark.parametrize("rows,topk,splits", [(1, 6, 0), (1, 6, 8), (3, 8, 9), (2, 9, 1), (5, 17, 20)])
def test_combine_of_routes_and_shared_planes(rows, topk, splits):
    """Around the number of routes and planes that are under way together, absent routes among them; same order, same bits."""
    from ds41rt_b200.ops import lib
    k = lib.kernels()
    torch.manual_seed(topk)
    H, active = 1028, 11
    fc2, shared = torch.randn(active, rows, H, device="cuda"), torch.randn(max(splits, 1), rows, H, device="cuda")
    slot = torch.randint(-1, active, (rows, topk), device="cuda", dtype=torch.int32)
    out = torch.full((rows, H), float("nan"), device="cuda")
    lib.check(k.ds41_moe_combine(lib.ptr(fc2), lib.ptr(slot), lib.ptr(shared), splits, rows, topk, H, lib.ptr(out), lib.stream()),
              "combine")
    want = torch.zeros(rows, H, device="cuda")
    for r in range(rows):
        for s in slot[r].tolist():
            if s >= 0:
                want[r] += fc2[s, r].bfloat16().float()
        for s in range(splits):
            want[r] += shared[s, r]
    assert torch.equal(out, want)


def test_quotient_against_the_division_operator():
    """v / s of the hyper-connection mixes over the pairs that they can meet and far beyond: the bits of the operator, which rounds
    correctly.  Zeros, powers of two and significands next to the end among them."""
    from ds41rt_b200.ops import lib
    n = 1 << 24
    g = torch.Generator(device="cuda").manual_seed(1)
    bits = lambda lo, hi: ((torch.randint(lo + 127, hi + 127, (n,), generator=g, device="cuda") << 23) |
                           torch.randint(0, 1 << 23, (n,), generator=g, device="cuda")).int()
    for v_range, s_range in (((-30, 1), (-20, 3)), ((0, 1), (0, 1)), ((-60, 60), (-60, 60))):
        v, s = bits(*v_range), bits(*s_range)
        v[::7] |= (1 << 23) - 1
        s[::11] |= (1 << 23) - 1
        s[5::11] &= ~((1 << 23) - 1)
        v, s = v.view(torch.float32), s.view(torch.float32)
        v[:8] = 0.0
        q = torch.full((n,), float("nan"), device="cuda")
        lib.check(lib.kernels().ds41_quotient(lib.ptr(v), lib.ptr(s), lib.ptr(q), C.c_longlong(n), lib.stream()), "quotient")
        assert torch.equal(q, v / s)
        assert float((q.double() * s.double() / v.double() - 1)[8:].abs().max()) <= 2.0 ** -24 * (1 + 2.0 ** -20)


@pytest.mark.parametrize("form", ["finish", "mixes"])
@pytest.mark.parametrize("spread", [0.5, 4.0, 12.0])
@pytest.mark.parametrize("iters", [1, 2, 20])
def test_mixes_against_64_bits(iters, spread, form):
    """The 4 x 4 matrix of every row.  A step divides a positive matrix by its row or column sums: in the logarithm of the ratios of
    its entries no step carries an error further than it found it, and each adds its own roundings (three additions, the
    divisor's, the quotient's and those of eps: 6 x 2^-24).  The exponentials are off by 2 units, and by their argument's
    rounding, |x| x 2^-23.  An entry is off by at most twice the largest of all that."""
    from ds41rt_b200.ops import lib
    k, rows, H, eps = lib.kernels(), 1000, 1024, 1e-6
    g = torch.Generator().manual_seed(iters)
    z = torch.randn(rows, 24, generator=g) * spread
    part = torch.zeros(1, rows, 25)
    part[0, :, :24], part[0, :, 24] = z, 4.0 * H                        # a row of unit size: its projections stand as they are
    part, planes = part.cuda(), torch.cat([z, torch.zeros(rows, 24)], 1).contiguous().cuda()
    scale, base = torch.ones(3).cuda(), torch.zeros(24).cuda()
    streams, pre_in = torch.randn(rows, 4, H, device="cuda").bfloat16(), torch.rand(rows, 4, device="cuda")
    pre, post, comb = torch.zeros(rows, 4).cuda(), torch.zeros(rows, 4).cuda(), torch.zeros(rows, 16).cuda()
    xn = torch.zeros(rows, H, device="cuda").bfloat16()
    finish = form == "finish"
    lib.check(k.ds41_hc_finish(lib.ptr(part), 1, lib.ptr(scale), lib.ptr(base), lib.ptr(pre_in), lib.ptr(streams), lib.ptr(None),
                               lib.ptr(pre), lib.ptr(post), lib.ptr(comb), lib.ptr(xn if finish else None), lib.ptr(None),
                               lib.ptr(None), lib.ptr(None), rows, H, iters, C.c_float(eps), C.c_float(0.0),
                               lib.ptr(None if finish else planes), 0 if finish else 1, C.c_longlong(rows * 48), 48, lib.stream()),
              "mixes")
    x = z[:, 8:].double().view(rows, 4, 4)
    want = torch.softmax(x, 2) + eps
    want = want / (want.sum(1, keepdim=True) + eps)
    for _ in range(iters - 1):
        want = want / (want.sum(2, keepdim=True) + eps)
        want = want / (want.sum(1, keepdim=True) + eps)
    reach = float((x.amax(2, keepdim=True) - x).max())
    bound = 2 * ((2 + 2 * reach) * 2.0 ** -23 + 2 * iters * 6 * 2.0 ** -24)
    off = float((comb.cpu().double().view(rows, 4, 4) / want - 1).abs().max())
    assert off <= bound
    assert float((pre.cpu().double() - (torch.sigmoid(z[:, :4].double()) + eps)).abs().max()) < 1e-5
    assert float((post.cpu().double() - 2 * torch.sigmoid(z[:, 4:8].double())).abs().max()) < 1e-5

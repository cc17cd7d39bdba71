"""tcgen05 GEMM kernel vs a plain PyTorch fp32 reference."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _ref(a, b):
    return a.float() @ b.float().t()


def _rel(out, ref):
    return float((out.float() - ref).abs().max() / ref.abs().max().clamp(min=1e-6))


@pytest.mark.parametrize("rows,N,K", [(1, 256, 512), (5, 1280, 5120), (16, 384, 1024), (64, 512, 192),
                                      (100, 640, 2304), (300, 1024, 512), (1000, 768, 1536), (300, 200, 512),
                                      (257, 72, 256)])
def test_matmul_nt_bf16(rows, N, K):
    from ds41rt_b200.ops import gemm as G, lib
    torch.manual_seed(rows + N)
    x = torch.randn(rows, K, device="cuda").bfloat16()
    w = (torch.randn(N, K, device="cuda") * 0.05).bfloat16()
    st = lib.new_status("cuda")
    out = G.matmul_nt(x, w, status=st)
    torch.cuda.synchronize()
    lib.raise_on_status(st, "gemm")
    assert _rel(out, _ref(x, w)) < 1e-2
    out32 = G.matmul_nt(x, w, out_dtype=torch.float32, status=st)
    torch.cuda.synchronize()
    assert _rel(out32, _ref(x, w)) < 2e-3


@pytest.mark.parametrize("rows,N,K,splits", [(4, 1792, 5120, 8), (8, 512, 1024, 4), (33, 384, 512, 2)])
def test_split_k_planes(rows, N, K, splits):
    from ds41rt_b200.ops import gemm as G, lib
    x = torch.randn(rows, K, device="cuda").bfloat16()
    w = (torch.randn(N, K, device="cuda") * 0.05).bfloat16()
    planes = torch.zeros(splits, rows, N, device="cuda")
    st = lib.new_status("cuda")
    G.linear_planes(x, w, planes, splits, status=st)
    torch.cuda.synchronize()
    lib.raise_on_status(st, "gemm split")
    assert _rel(planes.sum(0), _ref(x, w)) < 2e-3


def test_batched_grouped_output():
    """wo_a shape: per-group weights [G, o, k], activations [rows, G*k] -> [rows, G*o]."""
    from ds41rt_b200.ops import gemm as G, lib
    g, o, k, rows = 2, 256, 1024, 6
    w = (torch.randn(g, o, k, device="cuda") * 0.05).bfloat16()
    x = torch.randn(rows, g * k, device="cuda").bfloat16()
    out = torch.zeros(rows, g * o, device="cuda", dtype=torch.bfloat16)
    st = lib.new_status("cuda")
    G.gemm_raw(w, x, out, o, rows, k, lda=k, ldb=g * k, ldo=g * o, out_mode=2, batch=g, a_batch_stride=o * k,
               b_batch_stride=k, out_batch_stride=o, status=st)
    torch.cuda.synchronize()
    lib.raise_on_status(st, "gemm batched")
    ref = torch.einsum("rgk,gok->rgo", x.float().view(rows, g, k), w.float()).reshape(rows, g * o)
    assert _rel(out, ref) < 1e-2


def test_fp8_unscaled():
    from ds41rt_b200.ops import gemm as G, lib
    rows, N, K = 7, 512, 1024
    x = torch.randn(rows, K, device="cuda").to(torch.float8_e4m3fn)
    w = torch.randn(N, K, device="cuda").to(torch.float8_e4m3fn)
    out = torch.zeros(rows, N, device="cuda")
    st = lib.new_status("cuda")
    G.gemm_raw(w, x, out, N, rows, K, lda=K, ldb=K, ldo=N, kind=1, out_mode=3, status=st)
    torch.cuda.synchronize()
    lib.raise_on_status(st, "gemm fp8")
    assert _rel(out, _ref(x, w)) < 1e-3


@pytest.mark.parametrize("rows,N,K", [(5, 256, 512), (40, 384, 1024), (128, 256, 256), (300, 256, 512)])
def test_mxfp8_block_scaled(rows, N, K):
    from ds41rt_b200.ops import gemm as G, lib, quant_ref as Q
    from ds41rt_b200.ops.mx import pack_sf_atoms
    torch.manual_seed(1)
    x = torch.randn(rows, K, device="cuda") * torch.exp(torch.randn(rows, 1, device="cuda"))
    w = torch.randn(N, K, device="cuda") * 0.1 * torch.exp(torch.randn(N, 1, device="cuda"))
    xq, xe = Q.quant_mxfp8(x)
    wq, we = Q.quant_mxfp8(w)
    ref = Q.dequant_mxfp8(xq, xe) @ Q.dequant_mxfp8(wq, we).t()
    st = lib.new_status("cuda")
    out = torch.zeros(rows, N, device="cuda")
    sfx, sfw = pack_sf_atoms(xe), pack_sf_atoms(we)
    if rows <= 128:
        G.gemm_raw(wq, xq, out, N, rows, K, lda=K, ldb=K, ldo=N, kind=2, out_mode=3, sfa=sfw, sfb=sfx,
                   bn=max(32, G.pick_bn(rows)), status=st)
    else:
        G.gemm_raw(xq, wq, out, rows, N, K, lda=K, ldb=K, ldo=N, kind=2, out_mode=1, sfa=sfx, sfb=sfw, bn=128,
                   status=st)
    torch.cuda.synchronize()
    lib.raise_on_status(st, "gemm mx")
    assert _rel(out, ref) < 2e-3


@pytest.mark.parametrize("rows,N,K", [(5, 256, 512), (40, 384, 1024), (16, 4608, 5120)])
def test_mxfp4_weights_times_mxfp8_rows(rows, N, K):
    """E2M1 weights (two per byte, UE8M0 per 32) as the M operand of the block-scaled kind, E4M3 rows as N."""
    from ds41rt_b200.ops import gemm as G, lib, quant_ref as Q
    from ds41rt_b200.ops.mx import pack_sf_atoms
    torch.manual_seed(2)
    x = torch.randn(rows, K, device="cuda") * torch.exp(torch.randn(rows, 1, device="cuda"))
    w = torch.randn(N, K, device="cuda") * 0.1 * torch.exp(torch.randn(N, 1, device="cuda"))
    xq, xe = Q.quant_mxfp8(x)
    wq, we = Q.quant_mxfp4(w)
    ref = Q.dequant_mxfp8(xq, xe) @ Q.dequant_mxfp4(wq, we).t()
    st = lib.new_status("cuda")
    out = torch.zeros(rows, N, device="cuda")
    G.gemm_raw(wq.contiguous(), xq, out, N, rows, K, lda=K, ldb=K, ldo=N, kind=2, out_mode=3, sfa=pack_sf_atoms(we),
               sfb=pack_sf_atoms(xe), bn=max(32, G.pick_bn(rows)), status=st, a_format=1)
    torch.cuda.synchronize()
    lib.raise_on_status(st, "gemm mxfp4")
    assert _rel(out, ref) < 2e-3


@pytest.mark.parametrize("rows,N,K", [(5, 256, 512), (40, 384, 1024), (16, 4608, 5120), (300, 256, 768)])
def test_nvfp4_both_operands(rows, N, K):
    """E2M1 values with an E4M3 scale per 16 elements and one fp32 scale per tensor (NVFP4) on both operands:
    tcgen05 kind::mxf4nvf4, scale_vec 4X, global scales folded into the epilogue."""
    from ds41rt_b200.ops import gemm as G, lib, quant_ref as Q
    from ds41rt_b200.ops.mx import pack_sf_atoms
    torch.manual_seed(3)
    x = torch.randn(rows, K, device="cuda") * torch.exp(0.5 * torch.randn(rows, 1, device="cuda"))
    w = torch.randn(N, K, device="cuda") * 0.1 * torch.exp(0.5 * torch.randn(N, 1, device="cuda"))
    xq, xs, xg = Q.quant_nvfp4(x)
    wq, ws, wg = Q.quant_nvfp4(w)
    ref = Q.dequant_nvfp4(xq, xs, xg) @ Q.dequant_nvfp4(wq, ws, wg).t()
    st = lib.new_status("cuda")
    out = torch.zeros(rows, N, device="cuda")
    sfx = pack_sf_atoms(xs.view(torch.uint8))
    sfw = pack_sf_atoms(ws.view(torch.uint8))
    alpha = float(xg) * float(wg)
    if rows <= 128:
        G.gemm_raw(wq.contiguous(), xq.contiguous(), out, N, rows, K, lda=K, ldb=K, ldo=N, kind=3, out_mode=3, sfa=sfw,
                   sfb=sfx, bn=max(32, G.pick_bn(rows)), status=st, alpha=alpha)
    else:
        G.gemm_raw(xq.contiguous(), wq.contiguous(), out, rows, N, K, lda=K, ldb=K, ldo=N, kind=3, out_mode=1, sfa=sfx,
                   sfb=sfw, bn=128, status=st, alpha=alpha)
    torch.cuda.synchronize()
    lib.raise_on_status(st, "gemm nvfp4")
    assert _rel(out, ref) < 2e-3


@pytest.mark.parametrize("bn", [64, 128, 256])
def test_fp32_rows_of_a_tile_table_end_with_their_group(bn):
    """bf16 groups at any column, in one plane: columns between and behind the groups stay as they were, whatever the
    (unused) stride between batches."""
    import ctypes as C
    from ds41rt_b200.ops import lib
    g = torch.Generator().manual_seed(bn)
    E, M, K, cap = 3, 200, 320, 700
    groups = [(0, 37), (37, 37 + 150), (301, 301 + 257)]                 # first column, end
    x, w = torch.randn(cap, K, generator=g).bfloat16(), (torch.randn(E, M, K, generator=g) * 0.05).bfloat16()
    tiles = [(e, r, min(r + bn, b)) for e, (a, b) in enumerate(groups) for r in range(a, b, bn)]
    tab = torch.tensor(tiles + [(0, 0, cap)] * 2, dtype=torch.int32).T.contiguous().cuda()
    n = torch.tensor([len(tiles)], dtype=torch.int32).cuda()
    X, W, st = x.cuda(), w.cuda(), lib.new_status("cuda")
    out = torch.full((2 * M, cap), 7.0, device="cuda")                   # a plane more than the product has
    a = lib.GemmArgs()
    a.A, a.B, a.out, a.status = lib.ptr(W), lib.ptr(X), lib.ptr(out), lib.ptr(st)
    a.lda, a.ldb, a.ldo, a.M, a.N, a.K, a.batch, a.a_batches, a.a_batch_stride = K, K, cap, M, cap, K, E, E, M * K
    a.out_batch_stride, a.kind, a.out_mode, a.k_splits, a.b_batch_kind, a.bn = M * cap, 0, 1, 1, 1, bn
    a.tile_group, a.tile_row0, a.tile_end = (lib.ptr(t) for t in tab)
    a.n_tiles_dev, a.max_tiles = lib.ptr(n), len(tiles) + 2
    lib.check(lib.kernels().ds41_gemm_tc(C.byref(a), lib.stream()), "gemm")
    torch.cuda.synchronize()
    lib.raise_on_status(st, "gemm tile table")
    got, want, held = out.cpu(), torch.full((2 * M, cap), 7.0), torch.zeros(cap, dtype=torch.bool)
    for e, (c0, c1) in enumerate(groups):
        want[:M, c0:c1] = _ref(w[e], x[c0:c1])
        held[c0:c1] = True
    assert _rel(got[:M, held], want[:M, held]) < 2e-3
    assert bool((got[:, ~held] == 7.0).all()) and bool((got[M:] == 7.0).all())


def _swapped_and_wide(rows, N, K, seed=0):
    g = torch.Generator().manual_seed(rows + N + seed)
    x, w = torch.randn(rows, K, generator=g).bfloat16().cuda(), (torch.randn(N, K, generator=g) * 0.05).bfloat16().cuda()
    return x, w


@pytest.mark.parametrize("rows,N,K", [(129, 18944, 136), (333, 12676, 192), (333, 12801, 72), (1025, 4250, 320), (2049, 2306, 64)])
def test_planes_of_long_passes_are_those_of_the_swapped_form(rows, N, K):
    """Rows as the 128-row operand and 256 weight rows as the other one, stored by TMA where the rows allow it: the same products
    in the same order, bit for bit, at ragged rows, columns and depths."""
    from ds41rt_b200.ops import gemm as G, lib
    assert G.wide(rows, N) and not G.wide(128, 1 << 20) and not G.wide(rows, 256)
    x, w = _swapped_and_wide(rows, N, K)
    st = lib.new_status("cuda")
    flat = torch.full((rows * N + 64,), 7.0, device="cuda")
    planes = flat[: rows * N].view(1, rows, N)
    G.linear_planes(x, w, planes, 1, status=st)
    want = torch.zeros(rows, N, device="cuda")
    G.gemm_raw(w, x, want, N, rows, K, lda=K, ldb=K, ldo=N, out_mode=3, status=st)
    torch.cuda.synchronize()
    lib.raise_on_status(st, "gemm wide")
    assert torch.equal(planes[0], want) and bool((flat[rows * N:] == 7.0).all())
    assert _rel(want, _ref(x, w)) < 2e-3


@pytest.mark.parametrize("mode", [1, 6])
@pytest.mark.parametrize("rows,N,K,pad,batch", [(333, 1000, 192, 24, 1), (1025, 264, 128, 8, 1), (300, 200, 72, 0, 3), (129, 72, 64, 8, 4),
                                                (40, 328, 256, 0, 2)])
def test_stores_of_wide_forms_keep_to_their_columns(mode, rows, N, K, pad, batch):
    """fp32 and bf16 rows through TMA stores: longer output rows than the product has columns, and batches side by side in one
    row.  Bit for bit what the swapped form stores; what lies between stays as it was."""
    from ds41rt_b200.ops import gemm as G, lib
    g = torch.Generator().manual_seed(rows + mode)
    x = torch.randn(rows, batch * K, generator=g).bfloat16().cuda()
    w = (torch.randn(batch, N, K, generator=g) * 0.05).bfloat16().cuda()
    dt, ld, st = (torch.float32 if mode == 1 else torch.bfloat16), batch * (N + pad), lib.new_status("cuda")
    got, want = (torch.full((rows + 2, ld), 7.0, device="cuda", dtype=dt) for _ in range(2))
    G.gemm_raw(x, w, got, rows, N, K, lda=batch * K, ldb=K, ldo=ld, out_mode=mode, bn=256, batch=batch, a_batch_stride=K,
               b_batch_stride=N * K, out_batch_stride=N + pad, status=st, static_operand=2)
    G.gemm_raw(w, x, want, N, rows, K, lda=K, ldb=batch * K, ldo=ld, out_mode=3 if mode == 1 else 2, batch=batch,
               a_batch_stride=N * K, b_batch_stride=K, out_batch_stride=N + pad, status=st)
    torch.cuda.synchronize()
    lib.raise_on_status(st, "gemm wide")
    assert torch.equal(got, want)
    held = want.view(rows + 2, batch, N + pad)
    assert bool((held[rows:] == 7.0).all()) and bool((held[:, :, N:] == 7.0).all())
    ref = torch.einsum("rbk,bnk->rbn", x.float().view(rows, batch, K), w.float())
    assert _rel(held[:rows, :, :N], ref) < (2e-3 if mode == 1 else 1e-2)


def test_outputs_that_no_tensor_map_describes_take_plain_stores():
    """fp32 rows at odd lengths, off 16 bytes, and one row whose length says nothing."""
    from ds41rt_b200.ops import gemm as G, lib
    rows, N, K = 300, 72, 64
    x, w = _swapped_and_wide(rows, N, K)
    st = lib.new_status("cuda")
    ref = _ref(x, w)
    for ld, off, m in ((75, 0, rows), (76, 1, rows), (0, 0, 1)):
        flat = torch.full((rows * 80,), 7.0, device="cuda")
        G.gemm_raw(x, w, flat[off:], m, N, K, lda=K, ldb=K, ldo=ld, out_mode=1, bn=64, status=st)
        torch.cuda.synchronize()
        lib.raise_on_status(st, "gemm")
        step = max(ld, N)
        out = flat[off: off + m * step].view(m, step)
        assert _rel(out[:, :N], ref[:m]) < 2e-3 and bool((out[:, N:] == 7.0).all()) and bool((flat[off + m * step:] == 7.0).all())


def test_gathered_rows_of_one_rank_through_staged_stores():
    """The all-gather form with a world of one (no waits, no copies): the same rows as without it."""
    import ctypes as C
    from ds41rt_b200.ops import gemm as G, lib
    rows, N, K = 384, 200, 192
    x, w = _swapped_and_wide(rows, N, K)
    st = lib.new_status("cuda")
    got, want = torch.full((rows, 208), 7.0, device="cuda"), torch.full((rows, 208), 7.0, device="cuda")
    arrive, epoch = torch.zeros(8, dtype=torch.int32, device="cuda"), torch.ones(1, dtype=torch.int32, device="cuda")
    a = lib.GemmArgs()
    a.B, a.out, a.status = lib.ptr(w), lib.ptr(got), lib.ptr(st)
    a.lda, a.ldb, a.ldo, a.M, a.N, a.K, a.batch, a.a_batches = K, K, 208, rows, N, K, 1, 1
    a.kind, a.out_mode, a.k_splits, a.bn = 0, 1, 1, 128
    a.ag_world, a.ag_rank, a.ag_rows, a.ag_epoch = 1, 0, rows, lib.ptr(epoch)
    a.a_peers[0], a.ag_arrive[0] = x.data_ptr(), arrive.data_ptr()
    lib.check(lib.kernels().ds41_gemm_tc(C.byref(a), lib.stream()), "gemm")
    G.gemm_raw(w, x, want, N, rows, K, lda=K, ldb=K, ldo=208, out_mode=3, status=st)
    torch.cuda.synchronize()
    lib.raise_on_status(st, "gemm gathered")
    assert torch.equal(got, want)

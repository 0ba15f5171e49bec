"""Copies, casts and thin products at the sizes where their vectors, tiles and index splits end."""
import pytest
import torch

pytestmark = pytest.mark.gpu

from flexflow_train_b200.ops import kernels as K  # noqa: E402


def _randn(*shape, dtype=torch.bfloat16, seed=0):
    return torch.randn(*shape, generator=torch.Generator(device="cuda").manual_seed(seed), device="cuda").to(dtype)


@pytest.mark.parametrize("n", [1, 7, 8, 4099, 1 << 20])
@pytest.mark.parametrize("accumulate", [False, True])
@pytest.mark.parametrize("offset", [0, 1])
def test_cast_up(n, accumulate, offset):
    s = _randn(n + offset)[offset:]
    d = _randn(n + offset, dtype=torch.float32, seed=1)[offset:]
    want = s.float() + d if accumulate else s.float()
    K.cast(s, d, accumulate=accumulate)
    assert torch.equal(d, want)


@pytest.mark.parametrize("rows,cols", [(1, 8), (7, 1024), (64, 1024), (65, 264), (300, 256), (2048, 512), (64, 10), (4096, 1)])
def test_bias_gradient_of_few_rows(rows, cols):
    dy, y = _randn(rows, cols), _randn(rows, cols, seed=1)
    dz, db = torch.empty_like(dy), torch.empty(cols, device="cuda").bfloat16()
    scratch = torch.empty(K.bias_act_bwd_scratch(rows, cols), device="cuda")
    K.bias_act_bwd(dy, y, dz, db, scratch, "relu")
    want = dy * (y > 0)
    assert torch.equal(dz, want)
    ref = want.double().sum(0)
    # fp32 sums of `rows` terms, one bf16 rounding
    assert ((db.double() - ref).abs() <= ref.abs() * 2.0 ** -8 + want.double().abs().sum(0) * rows * 2.0 ** -24 + 1e-7).all()


@pytest.mark.parametrize("rows,cols", [(1, 1), (7, 10), (64, 1024), (300, 33), (4096, 128), (4096, 256), (2048, 2056)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_bias_gradient_chunks(rows, cols, dtype):
    """Scalar and vector forms, whose rows are split differently, in the scratch one function reports for both."""
    dy = _randn(rows, cols, dtype=dtype)
    n = K.bias_act_bwd_scratch(rows, cols)
    scratch, db, old = torch.full((n + 64,), 7.0, device="cuda"), _randn(cols, dtype=dtype, seed=2), _randn(cols, dtype=dtype, seed=2)
    K.bias_act_bwd(dy, None, None, db, scratch[:n], None, accumulate=True)
    ref = dy.double().sum(0) + old.double()
    ulp = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -23
    assert ((db.double() - ref).abs() <= ref.abs() * ulp + (dy.double().abs().sum(0) + 1) * rows * 2.0 ** -24).all()
    assert (scratch[n:] == 7).all()


def test_bias_gradient_refuses_a_short_scratch():
    dy, db = _randn(800, 768), torch.zeros(768, device="cuda").bfloat16()
    short = torch.empty(K.bias_act_bwd_scratch(800, 768) - 1, device="cuda")
    for scratch in (short, None):
        with pytest.raises(K.KernelError, match="scratch"):
            K.bias_act_bwd(dy, None, None, db, scratch, None)
    K.bias_act_bwd(dy, _randn(800, 768, seed=1), torch.empty_like(dy), None, None, "relu")  # without a bias gradient none is needed


@pytest.mark.parametrize("dtype", [torch.uint8, torch.bfloat16, torch.float32, torch.int64])
@pytest.mark.parametrize("outer,block,src_ld,dst_ld,offset", [(1, 1, 1, 1, 0), (64, 5270, 5270, 5272, 0), (9, 13, 13, 16, 1), (257, 6, 9, 8, 2),
                                                              (5000, 942, 1000, 944, 3)])
def test_block_copy(dtype, outer, block, src_ld, dst_ld, offset):
    src = (torch.rand(outer * src_ld + offset, device="cuda") * 200).to(dtype)
    dst = torch.zeros(outer * dst_ld + offset, device="cuda", dtype=dtype)
    want = dst.clone()
    want[offset:].view(outer, dst_ld)[:, :block] = src[offset:].view(outer, src_ld)[:, :block]
    K.block_copy(src, offset, src_ld, dst, offset, dst_ld, outer, block)
    assert torch.equal(dst, want)


@pytest.mark.parametrize("shape,perm", [((4096, 9, 64), (0, 2, 1)), ((3, 5, 7, 11), (3, 1, 0, 2)), ((1, 1), (1, 0)), ((2, 3, 2, 3, 2, 3), (5, 3, 1, 4, 2, 0)),
                                        ((70000,), (0,))])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32, torch.int64])
def test_permute(shape, perm, dtype):
    x = (_randn(*shape, dtype=torch.float32) * 100).to(dtype)
    assert torch.equal(K.permute(x, perm), x.permute(perm).contiguous())
    if dtype != torch.int64:
        out = torch.ones_like(x.permute(perm).contiguous())
        K.permute(x, perm, out=out, accumulate=True)
        assert torch.equal(out, 1 + x.permute(perm))


@pytest.mark.parametrize("M,N,Kd", [(1, 1, 1), (64, 512, 10), (10, 512, 64), (17, 65, 33), (33, 7, 128), (100, 30, 129), (64, 2048, 3)])
@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float32])
def test_thin_products(M, N, Kd, dt):
    """Row pitches that TMA cannot address; K on both sides of the thin kernel's limit, with epilogue and batches."""
    a, b = _randn(2, M, Kd, dtype=dt), _randn(2, N, Kd, dtype=dt, seed=1)
    bias, old = _randn(N, dtype=dt, seed=2), _randn(2, M, N, dtype=dt, seed=3)
    ref = a.double() @ b.double().transpose(1, 2)
    tol = lambda w: Kd * 2.0 ** -20 + w.abs() * (2.0 ** -8 if dt == torch.bfloat16 else 2.0 ** -20) + 1e-6  # noqa: E731  fp32 sums, one rounding
    for a_mn in (False, True):
        for b_mn in (False, True):
            x, w = (a.transpose(1, 2).contiguous() if a_mn else a), (b.transpose(1, 2).contiguous() if b_mn else b)
            if a.element_size() * x.shape[2] % 16 == 0 and b.element_size() * w.shape[2] % 16 == 0 and Kd > 8:
                continue  # both addressable: the tensor cores' case
            C = old.clone()
            K.gemm_raw(M=M, N=N, K=Kd, A=x.data_ptr(), lda=x.shape[2], a_sb=M * Kd, a_mn=a_mn, B=w.data_ptr(), ldb=w.shape[2], b_sb=N * Kd,
                       b_mn=b_mn, C=C.data_ptr(), ldc=N, c_sb=M * N, nb=2, es=a.element_size(), out_fp32=dt == torch.float32,
                       bias=bias.data_ptr(), act=K.ACT_CODES["relu"], accumulate=True)
            want = torch.relu(ref + bias.double()) + old.double()
            assert ((C.double() - want).abs() <= tol(want)).all(), (a_mn, b_mn, (C.double() - want).abs().max().item())


@pytest.mark.parametrize("cols", [256, 512, 768, 1024, 1280])
@pytest.mark.parametrize("rows", [63, 64, 65, 2401])
@pytest.mark.parametrize("acc", [False, True])
def test_layernorm_backward_rows(rows, cols, acc):
    """Row counts around the blocks of the one-warp-per-row kernel (1280 columns take the block-per-row one)."""
    x, dy, g = _randn(rows, cols), _randn(rows, cols, seed=1), _randn(cols, seed=2)
    mean, rstd, y = torch.empty(rows, device="cuda"), torch.empty(rows, device="cuda"), torch.empty_like(x)
    K.layernorm_fwd(x, g, g, 1e-5, out=y, mean=mean, rstd=rstd)
    old, old2 = _randn(rows, cols, seed=3), _randn(rows, cols, seed=4)
    dx, dx2, dg, db = old.clone(), old2.clone(), _randn(cols, seed=5), _randn(cols, seed=6)
    og, ob = dg.clone(), db.clone()
    K.layernorm_bwd(dy, x, g, mean, rstd, dx, dg, db, torch.empty(K.layernorm_bwd_scratch(rows, cols), device="cuda"), accumulate_dx=acc,
                    accumulate_params=acc, dx2=dx2, accumulate_dx2=not acc)
    xd = x.double().requires_grad_(True)
    gd, bd = g.double().requires_grad_(True), g.double().requires_grad_(True)
    torch.nn.functional.layer_norm(xd, (cols,), gd, bd, 1e-5).backward(dy.double())

    def near(got, want, slack):
        assert ((got.double() - want).abs() <= want.abs() * 2.0 ** -8 + slack).all(), (got.double() - want).abs().max().item()

    # fp32 statistics and row sums against fp64: a few ulps of values of order |dy| * |gamma| * rstd
    near(dx, xd.grad + (old.double() if acc else 0), 1e-4)
    near(dx2, xd.grad + (0 if acc else old2.double()), 1e-4)
    sums = rows * 2.0 ** -24 * 16
    near(dg, gd.grad + (og.double() if acc else 0), sums * rows ** 0.5 + 1e-3)
    near(db, bd.grad + (ob.double() if acc else 0), sums * rows ** 0.5 + 1e-3)


def test_scatter_into_one_row():
    """Every token of every bag at the same row: whole numbers below 2^24, so that the sums are exact in any order."""
    for dim in (8, 64, 768):
        dout = torch.randint(-3, 4, (500, dim), device="cuda").float()
        idx = torch.full((500, 3), 17, device="cuda", dtype=torch.int64)
        table = torch.zeros(40, dim, device="cuda")
        K.embedding_bwd(idx, dout, table)
        assert torch.equal(table[17], 3 * dout.sum(0)) and not table[:17].any() and not table[18:].any()
        K.embedding_sgd(idx, dout.bfloat16(), table, 1.0)
        assert not table.any()


@pytest.mark.parametrize("dim", [8, 64, 2048, 12])
@pytest.mark.parametrize("bag,aggr", [(1, "sum"), (3, "sum"), (4, "avg")])
@pytest.mark.parametrize("table_dt,out_dt", [(torch.bfloat16, torch.bfloat16), (torch.float32, torch.bfloat16), (torch.float32, torch.float32)])
@pytest.mark.parametrize("idx_dt", [torch.int32, torch.int64])
def test_embedding_pieces(dim, bag, aggr, table_dt, out_dt, idx_dt):
    """Lookup, scatter and sparse step in 16-byte pieces (12 columns: element by element); indexes out of range count as nothing."""
    tokens, entries = 301, 1000
    table = _randn(entries, dim, dtype=torch.float32).to(table_dt)
    idx = torch.randperm(tokens * bag + 50, device="cuda", generator=torch.Generator(device="cuda").manual_seed(1))[:tokens * bag] % (entries + 1)
    idx = torch.where(idx == entries, -1, idx).to(idx_dt).view(tokens, bag)
    if bag > 1:
        out = torch.empty(tokens, dim, device="cuda", dtype=out_dt)
    else:
        out = torch.empty(tokens, 1, dim, device="cuda", dtype=out_dt).view(tokens, dim)
    K.embedding_fwd(idx, table, out, aggr=aggr)
    ok = (idx >= 0).double()[..., None]
    rows = table.double()[idx.long().clamp(min=0)] * ok
    want = rows.sum(1) / (bag if aggr == "avg" else 1)
    ulp = lambda dt: 2.0 ** -8 if dt == torch.bfloat16 else 2.0 ** -22  # noqa: E731
    assert ((out.double() - want).abs() <= want.abs() * ulp(out_dt) + rows.abs().sum(1) * 2.0 ** -22).all()
    dout = _randn(tokens, dim, dtype=torch.float32, seed=2).to(out_dt)
    dt = torch.zeros_like(table)
    K.embedding_bwd(idx, dout, dt, aggr=aggr)
    ref = torch.zeros(entries, dim, device="cuda", dtype=torch.float64)
    mag = torch.zeros_like(ref)
    g = (dout.double() / (bag if aggr == "avg" else 1))[:, None].expand(-1, bag, -1) * ok
    ref.index_put_((idx.long().clamp(min=0).view(-1),), g.reshape(-1, dim), accumulate=True)
    mag.index_put_((idx.long().clamp(min=0).view(-1),), g.abs().reshape(-1, dim), accumulate=True)
    assert ((dt.double() - ref).abs() <= mag * 4 * ulp(table_dt)).all()  # at most a few additions per row, one rounding each
    if table_dt == torch.float32:
        t2 = table.clone()
        K.embedding_sgd(idx, dout, t2, 0.5, aggr=aggr)
        assert ((t2.double() - (table.double() - 0.5 * ref)).abs() <= (mag + table.double().abs()) * 2.0 ** -20).all()


@pytest.mark.parametrize("cols", [256, 512, 768, 1024, 1280])
@pytest.mark.parametrize("rows", [7, 64, 1201])
def test_layernorm_fp32_rows(rows, cols):
    x, r, dy, g, b = (_randn(*s, dtype=torch.float32, seed=i) for i, s in enumerate([(rows, cols), (rows, cols), (rows, cols), (cols,), (cols,)]))
    mean, rstd, y, xsum = torch.empty(rows, device="cuda"), torch.empty(rows, device="cuda"), torch.empty_like(x), torch.empty_like(x)
    K.layernorm_fwd(x, g, b, 1e-5, residual=r, xsum=xsum, out=y, mean=mean, rstd=rstd)
    assert torch.equal(xsum, x + r)
    xd, gd, bd = xsum.double().requires_grad_(True), g.double().requires_grad_(True), b.double().requires_grad_(True)
    ref = torch.nn.functional.layer_norm(xd, (cols,), gd, bd, 1e-5)
    # fp32 row sums of `cols` terms of order one, combined in a tree of depth log2(cols) + 8
    eps = 2.0 ** -24 * 32
    assert (y.double() - ref).abs().max() <= 8 * eps * ref.abs().max()
    ref.backward(dy.double())
    dx, dg, db = torch.empty_like(x), torch.empty_like(g), torch.empty_like(b)
    K.layernorm_bwd(dy, xsum, g, mean, rstd, dx, dg, db, torch.empty(K.layernorm_bwd_scratch(rows, cols), device="cuda"))
    assert (dx.double() - xd.grad).abs().max() <= 8 * eps * xd.grad.abs().max()
    for got, want in ((dg, gd.grad), (db, bd.grad)):
        assert (got.double() - want).abs().max() <= 8 * eps * max(want.abs().max().item(), rows ** 0.5)


@pytest.mark.parametrize("M,N,Kd", [(9, 9, 64), (9, 64, 9), (64, 9, 9), (1, 1, 5), (5, 33, 20)])
@pytest.mark.parametrize("out_dt", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("accumulate", [False, True])
def test_small_batched_products(M, N, Kd, out_dt, accumulate):
    a, b, old = _randn(70, M, Kd), _randn(70, N, Kd, seed=1), _randn(70, M, N, dtype=torch.float32, seed=2).to(out_dt)
    C = old.clone()
    K.gemm_raw(M=M, N=N, K=Kd, A=a.data_ptr(), lda=Kd, a_sb=M * Kd, B=b.data_ptr(), ldb=Kd, b_sb=N * Kd, C=C.data_ptr(), ldc=N, c_sb=M * N,
               nb=70, alpha=0.5, out_fp32=out_dt == torch.float32, accumulate=accumulate)
    want = 0.5 * (a.double() @ b.double().transpose(1, 2)) + (old.double() if accumulate else 0)
    ulp = 2.0 ** -8 if out_dt == torch.bfloat16 else 0
    assert ((C.double() - want).abs() <= want.abs() * ulp + Kd * 2.0 ** -20).all()  # fp32 sums of Kd terms, one rounding


@pytest.mark.parametrize("n", [1, 3, 4, 1021, 4096, 148 * 8 * 256 * 8 + 6])
@pytest.mark.parametrize("grad_dt", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("offset", [0, 1])  # 1: gradients that no 8- or 16-byte load takes (SGD: no array is aligned)
def test_optimizer_steps(n, grad_dt, offset):
    g = _randn(n + offset, dtype=torch.float32).to(grad_dt)[offset:]
    w, m, v = _randn(n, dtype=torch.float32, seed=1), _randn(n, dtype=torch.float32, seed=2), _randn(n, dtype=torch.float32, seed=3).abs()
    wd, md, vd, gd = w.double(), m.double(), v.double(), g.double()
    shadow = torch.zeros(n, device="cuda").bfloat16()
    K.adam_update(w, m, v, g, shadow, 1e-2, 0.9, 0.99, 1e-8, weight_decay=0.1)
    gt = gd + 0.1 * wd
    md = 0.9 * md + (1 - 0.9) * gt
    vd = 0.99 * vd + (1 - 0.99) * gt * gt
    want = wd - 1e-2 * md / (vd.sqrt() + 1e-8)
    # single-precision steps with approximate division and square root (2 ulp each) of values of order one
    for got, ref in ((m, md), (v, vd), (w, want)):
        assert ((got.double() - ref).abs() <= 2.0 ** -20 * (1 + ref.abs())).all()
    assert torch.equal(shadow, w.bfloat16())
    for momentum, nesterov in ((0.0, False), (0.9, False), (0.9, True)):
        w = _randn(n + offset, dtype=torch.float32, seed=4)[offset:]
        mom = _randn(n + offset, dtype=torch.float32, seed=5)[offset:] if momentum else None
        shadow = torch.zeros(n + offset, device="cuda").bfloat16()[offset:]
        gt = gd + 0.1 * w.double()
        ref_m = mom.double() * momentum + gt if momentum else None
        step = gt if not momentum else gt + momentum * ref_m if nesterov else ref_m
        want = w.double() - 0.05 * step
        K.sgd_update(w, mom, g, shadow, 0.05, momentum=momentum, nesterov=nesterov, weight_decay=0.1)
        assert ((w.double() - want).abs() <= 2.0 ** -20 * (1 + want.abs())).all()
        if momentum:
            assert ((mom.double() - ref_m).abs() <= 2.0 ** -20 * (1 + ref_m.abs())).all()
        assert torch.equal(shadow, w.bfloat16())

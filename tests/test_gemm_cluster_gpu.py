"""GEMM whose K range is shared by a cluster, at the edges of its tiles and with every epilogue, against fp64."""
import pytest
import torch

pytestmark = pytest.mark.gpu

from flexflow_train_b200.ops import kernels as K  # noqa: E402


def _operands(M, N, Kd, a_mn, b_mn, dt, batch=1):
    g = torch.Generator(device="cuda").manual_seed(M * 7 + N * 3 + Kd)
    pad = 16 // dt.itemsize
    up = lambda n: (n + pad - 1) // pad * pad  # noqa: E731  TMA wants row pitches of 16 bytes
    a = torch.randn(batch, Kd if a_mn else M, up(M if a_mn else Kd), generator=g, device="cuda").to(dt)
    b = torch.randn(batch, Kd if b_mn else N, up(N if b_mn else Kd), generator=g, device="cuda").to(dt)
    al = (a[:, :, :M].transpose(1, 2) if a_mn else a[:, :, :Kd]).double()
    bl = (b[:, :, :N].transpose(1, 2) if b_mn else b[:, :, :Kd]).double()
    return a, b, al @ bl.transpose(1, 2)


def _run(a, b, M, N, Kd, a_mn, b_mn, C, **kw):
    K.gemm_raw(M=M, N=N, K=Kd, A=a.data_ptr(), lda=a.shape[2], a_sb=a.stride(0), a_mn=a_mn, B=b.data_ptr(), ldb=b.shape[2],
               b_sb=b.stride(0), b_mn=b_mn, C=C.data_ptr(), es=a.element_size(), nb=a.shape[0], out_fp32=C.dtype == torch.float32, **kw)


def _close(got, want, scale, dt):
    # operands are exact in fp64; fp32 sums of Kd products (tf32 operands: 2^-11 each), then one rounding of the output
    slack = scale * (2.0 ** -9 if dt == torch.float32 else 2.0 ** -18) + want.abs() * (2.0 ** -8 if got.dtype == torch.bfloat16 else 0) + 1e-5
    bad = (got.double() - want).abs() > slack
    assert not bad.any(), (int(bad.sum()), (got.double() - want).abs().max().item())


SHAPES = [(1, 8, 128), (64, 10, 129), (127, 65, 512), (128, 64, 1000), (129, 130, 520), (300, 200, 2048)]


@pytest.mark.parametrize("M,N,Kd", SHAPES)
@pytest.mark.parametrize("order", ["nt", "nn", "tn", "tt"])
@pytest.mark.parametrize("bn,split", [(64, 2), (64, 8), (128, 2), (128, 4), (128, 8)])
def test_orders_and_edges(M, N, Kd, order, bn, split):
    if split > (Kd + 63) // 64:
        with pytest.raises(K.KernelError):
            a, b, _ = _operands(M, N, Kd, False, False, torch.bfloat16)
            _run(a, b, M, N, Kd, False, False, torch.empty(M, N, device="cuda", dtype=torch.bfloat16), ldc=N, bn=bn, split=split)
        return
    a_mn, b_mn = order[0] == "t", order[1] == "n"
    a, b, ref = _operands(M, N, Kd, a_mn, b_mn, torch.bfloat16)
    for dt in (torch.bfloat16, torch.float32):
        C = torch.full((M, N), 7.0, device="cuda", dtype=dt)
        _run(a, b, M, N, Kd, a_mn, b_mn, C, ldc=N, bn=bn, split=split)
        _close(C, ref[0], Kd, torch.bfloat16)
        again = torch.empty_like(C)
        _run(a, b, M, N, Kd, a_mn, b_mn, again, ldc=N, bn=bn, split=split)
        assert torch.equal(C, again)  # the partial sums are added in a fixed order
    assert K.gemm_last_error() == 0


@pytest.mark.parametrize("bn,split", [(64, 2), (64, 4), (128, 8)])
@pytest.mark.parametrize("N", [64, 67])
@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float32])
def test_epilogues(bn, split, N, dt):
    M, Kd = 150, 576
    a, b, ref = _operands(M, N, Kd, False, False, dt, batch=2)
    g = torch.Generator(device="cuda").manual_seed(5)
    bias = torch.randn(N, generator=g, device="cuda").to(dt)
    add = torch.randn(2, M, N, generator=g, device="cuda").to(dt)
    old = torch.randn(2, M, N, generator=g, device="cuda").to(dt)
    C, pre = old.clone(), torch.empty_like(old)
    _run(a, b, M, N, Kd, False, False, C, ldc=N, c_sb=M * N, bn=bn, split=split, alpha=0.5, bias=bias.data_ptr(), act=K.ACT_CODES["gelu"],
         C2=pre.data_ptr(), addend=add.data_ptr(), ld_add=N, add_sb=M * N, accumulate=True)
    z = ref * 0.5 + bias.double()
    _close(pre, z, Kd, dt)
    want = torch.nn.functional.gelu(z) + add.double() + old.double()
    _close(C, want, Kd, dt)
    C = torch.empty_like(old)
    _run(a, b, M, N, Kd, False, False, C, ldc=N, c_sb=M * N, bn=bn, split=split, bias=bias.data_ptr(), act=K.ACT_CODES["relu"])
    _close(C, torch.relu(ref + bias.double()), Kd, dt)


@pytest.mark.parametrize("M,N,Kd", [(64, 512, 784), (2048, 512, 512), (2048, 512, 4096), (1000, 3072, 768), (256, 512, 4096), (37, 1000, 2048)])
@pytest.mark.parametrize("accumulate", [False, True])
def test_chosen_kernel(M, N, Kd, accumulate):
    """Sizes on both sides of the rule that picks tile and kernel."""
    a, b, ref = _operands(M, N, Kd, False, True, torch.bfloat16)
    old = torch.randn(M, N, device="cuda").bfloat16()
    C = old.clone()
    _run(a, b, M, N, Kd, False, True, C, ldc=N, accumulate=accumulate)
    _close(C, ref[0] + (old.double() if accumulate else 0), Kd, torch.bfloat16)
    assert K.gemm_last_error() == 0


@pytest.mark.parametrize("M,N,Kd", [(4, 8, 4), (64, 96, 36), (128, 64, 512), (130, 132, 200), (300, 260, 1000), (2048, 512, 4096), (512, 512, 37), (20, 24, 7)])
def test_fp32_transposed_operands(M, N, Kd):
    """tf32 products that read their operands as they lie give what they give on transposed copies."""
    g = torch.Generator(device="cuda").manual_seed(M + N + Kd)
    a, b = torch.randn(M, Kd, generator=g, device="cuda"), torch.randn(N, Kd, generator=g, device="cuda")
    ref = a.double() @ b.double().t()
    at, bt = a.t().contiguous(), b.t().contiguous()
    for got in (K.matmul_nt(a, b), K.matmul_nn(a, bt), K.matmul_tn(at, bt)):
        # operands cut to 11 bits (2^-10 relative each), errors of random sign: far below Kd^0.5 * 6 of them
        assert (got.double() - ref).abs().max() <= 6 * Kd ** 0.5 * 2.0 ** -9
    old = torch.randn(M, N, generator=g, device="cuda")
    c = old.clone()
    K.matmul_tn(at, bt, out=c, accumulate=True)
    assert (c.double() - old.double() - ref).abs().max() <= 6 * Kd ** 0.5 * 2.0 ** -9
    if Kd % 4:  # small or repacked: no further from fp64 than the transposed copies were
        assert (K.matmul_tn(at, bt).double() - ref).norm() <= 1.01 * (K.matmul_nt(a, b).double() - ref).norm() + 1e-6
    assert K.gemm_last_error() == 0


@pytest.mark.parametrize("M,N", [(64, 192), (256, 512), (512, 512), (768, 768), (1000, 300)])
@pytest.mark.parametrize("Kd", [1024, 4096, 8192, 16384])
def test_fp32_results_keep_their_accumulators_short(M, N, Kd):
    """The chosen kernel's fp32 result is no further from fp64 than that of the split the persistent kernel makes."""
    g = torch.Generator(device="cuda").manual_seed(M + N + Kd)
    a, b = torch.randn(Kd, M, generator=g, device="cuda").bfloat16(), torch.randn(Kd, N, generator=g, device="cuda").bfloat16()
    ref = a.double().t() @ b.double()
    off = lambda c: ((c.double() - ref).norm() / ref.norm()).item()  # noqa: E731
    out = torch.empty(M, N, device="cuda")
    chosen, split = off(K.matmul_tn(a, b, out=out)), off(K.matmul_tn(a, b, out=torch.empty_like(out), bn=128))
    # errors of 1e4 and more elements average out: the ratio is that of the ranges, which are whole k-blocks
    assert chosen <= 1.05 * split, (chosen, split)

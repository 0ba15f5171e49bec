"""One-pass softmax, softmax + dropout and softmax + cross-entropy at the row lengths where their vectors end."""
import pytest
import torch

pytestmark = pytest.mark.gpu

from flexflow_train_b200.ops import kernels as K  # noqa: E402

# a bf16 result is within half an ulp (2^-9) of a value that carries the fp32 exponential's error (|x| * 2^-23 and 2 ulp)
REL = 2.0 ** -8


def _near(got, want, floor=1e-8):
    want = want.double()
    bad = (got.double() - want).abs() > REL * want.abs() + floor
    assert not bad.any(), (int(bad.sum()), (got.double() - want).abs().max().item())


@pytest.mark.parametrize("cols", [8, 248, 256, 264, 1000, 4088, 4096, 4104, 8192, 8200, 32000, 32776, 65536, 65544])
@pytest.mark.parametrize("rows", [5, 700])  # 700: more rows than blocks, every ring stage is filled again
def test_softmax_and_cross_entropy_rows(cols, rows):
    gen = torch.Generator(device="cuda").manual_seed(cols)
    x = (torch.randn(rows, cols, generator=gen, device="cuda") * 3).bfloat16()
    x[1, 0], x[2, cols - 1] = float("-inf"), 40.0  # a masked logit, a row whose last element dominates
    ref = torch.softmax(x.double(), -1)
    _near(K.softmax_fwd(x), ref)
    _near(K.softmax_fwd(x, scale=0.25), torch.softmax(x.double() * 0.25, -1))
    for dt in (torch.int32, torch.int64):
        labels = torch.randint(0, cols, (rows,), generator=gen, device="cuda", dtype=dt)
        labels[:4] = torch.tensor([0, cols - 1, cols - 1, -1], device="cuda", dtype=dt)
        loss, dl, probs = torch.empty(rows, device="cuda"), torch.empty_like(x), torch.empty_like(x)
        K.softmax_ce(x, labels, loss, dl, probs, grad_scale=0.5)
        _near(probs, ref)
        want = ref.clone()
        want[torch.arange(rows, device="cuda"), labels.long().clamp(min=0)] -= 1
        want[3] = 0
        _near(dl, want * 0.5, floor=2.0 ** -22)  # p - 1 cancels: fp32 ulps of 1
        wl = torch.logsumexp(x.double(), -1) - x.double().gather(1, labels.long().clamp(min=0)[:, None])[:, 0]
        wl[3] = 0
        assert torch.allclose(loss.double(), wl, rtol=1e-5, atol=1e-5)
    assert K.softmax_last_error() == 0


@pytest.mark.parametrize("cols", [1536, 1544, 2040, 2048, 2056, 4088, 4096])
@pytest.mark.parametrize("causal", [False, True])
def test_rows_on_both_sides_of_the_warp_kernels(cols, causal):
    """Plain softmax, forward and backward, where rows change from one warp each to one block each."""
    gen = torch.Generator(device="cuda").manual_seed(cols)
    x, dy = (torch.randn(70, cols, generator=gen, device="cuda").bfloat16() for _ in range(2))
    xd = x.double() * 0.5
    if causal:
        xd = xd.masked_fill(torch.arange(cols, device="cuda")[None] > (torch.arange(70, device="cuda") % 35)[:, None], float("-inf"))
    ref = torch.softmax(xd, -1)
    y, y2, dx, dx2 = (torch.empty_like(x) for _ in range(4))
    K.softmax_fwd(x, out=y, scale=0.5, causal_q=35 if causal else 0)
    K.softmax_dropout_fwd(x, y2, None, 0.0, 1, None, scale=0.5, causal_q=35 if causal else 0)
    _near(y, ref)
    assert torch.equal(y, y2)
    K.softmax_bwd(dy, y, dx=dx, scale=0.5)
    K.softmax_dropout_bwd(dy, y, dx2, 0.0, 1, None, scale=0.5)
    g, yr = dy.double(), y.double()
    want = 0.5 * yr * (g - (g * yr).sum(-1, keepdim=True))
    slack = 0.5 * yr * (g * yr).abs().sum(-1, keepdim=True) * cols * 2.0 ** -24
    assert ((dx.double() - want).abs() <= REL * want.abs() + slack + 1e-9).all() and torch.equal(dx, dx2)


@pytest.mark.parametrize("cols", [264, 4096, 4104, 16384, 16392, 32768, 32776])
def test_loss_alone(cols):
    """Cross-entropy without gradient or probabilities."""
    x = torch.randn(300, cols, generator=torch.Generator(device="cuda").manual_seed(cols), device="cuda").bfloat16()
    labels = torch.arange(300, device="cuda", dtype=torch.int32) * 7 % cols
    labels[5] = -1
    loss = torch.empty(300, device="cuda")
    K.softmax_ce(x, labels, loss)
    want = torch.logsumexp(x.double(), -1) - x.double().gather(1, labels.long().clamp(min=0)[:, None])[:, 0]
    want[5] = 0
    assert torch.allclose(loss.double(), want, rtol=1e-5, atol=1e-5)


@pytest.mark.parametrize("cols", [4096, 8192, 32776, 65544, 131072])
def test_rows_with_masked_pieces(cols):
    """Whole pieces, and a thread's and a warp's whole share of the row, masked out."""
    x = torch.randn(6, cols, generator=torch.Generator(device="cuda").manual_seed(cols), device="cuda").bfloat16()
    x[0, :8], x[1, 8:], x[2, :cols - 8], x[3, : cols // 2] = (float("-inf"),) * 4
    ref = torch.softmax(x.double(), -1)
    _near(K.softmax_fwd(x), ref)
    labels = torch.tensor([9, 3, cols - 1, cols - 2, 0, -1], device="cuda")
    loss, probs = torch.empty(6, device="cuda"), torch.empty_like(x)
    K.softmax_ce(x, labels, loss, x, probs)  # the gradient in the place of the logits
    _near(probs, ref)
    want = -torch.log(ref.gather(1, labels.clamp(min=0)[:, None]))[:, 0]
    want[5] = 0
    assert torch.allclose(loss.double(), want, rtol=1e-5, atol=1e-5)


@pytest.mark.parametrize("rows,cols", [(5, 4104), (700, 8192), (300, 32768)])
def test_rows_given_up_hold_no_numbers(rows, cols):
    """A wait that runs out must not leave an earlier call's values in the place of results."""
    x = torch.randn(rows, cols, device="cuda").bfloat16()
    labels = torch.zeros(rows, device="cuda", dtype=torch.int32)
    loss, dl, probs = torch.ones(rows, device="cuda"), torch.ones_like(x), torch.ones_like(x)
    K.softmax_ce_wait(x, labels, loss, dl, probs, 0)
    assert K.softmax_last_error() != 0 and K.softmax_last_error() == 0  # read and cleared
    assert loss.isnan().all() and dl.isnan().all() and probs.isnan().all()
    K.softmax_ce_wait(x, labels, loss, dl, probs, 10**9)
    _near(probs, torch.softmax(x.double(), -1))
    assert K.softmax_last_error() == 0 and loss.isfinite().all() and dl.isfinite().all()


@pytest.mark.skipif(torch.cuda.device_count() < 2, reason="needs two GPUs")
def test_wide_rows_on_every_device_of_a_process():
    for dev in range(2):
        with torch.cuda.device(dev):
            x = torch.randn(3, 8192, device="cuda").bfloat16()
            _near(K.softmax_fwd(x), torch.softmax(x.double(), -1))


def test_vocabularies_beyond_the_ring_keep_its_rate():
    """The same number of elements in rows of 131072 as in rows of 32768: a scalar form of the long rows takes several times as long."""
    def us(rows, cols, fn):
        x = torch.randn(rows, cols, device="cuda").bfloat16()
        labels = torch.zeros(rows, device="cuda", dtype=torch.int32)
        loss, dl = torch.empty(rows, device="cuda"), torch.empty_like(x)
        got = []
        for _ in range(8):
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record()
            K.softmax_ce(x, labels, loss, dl) if fn == "ce" else K.softmax_fwd(x, out=dl)
            e1.record()
            e1.synchronize()
            got.append(e0.elapsed_time(e1))
        return sorted(got)[3]

    for fn in ("ce", "softmax"):
        assert us(1024, 131072, fn) < 2.5 * us(4096, 32768, fn), fn


@pytest.mark.parametrize("cols", [1, 7, 9, 250, 255, 257, 500, 1001, 4090])
@pytest.mark.parametrize("causal", [False, True])
def test_pitched_softmax_dropout(cols, causal):
    gen = torch.Generator(device="cuda").manual_seed(cols)
    rows, ld = 37, K.softmax_pitch(cols)
    seed, salt, p = torch.tensor([1234567], device="cuda"), 99, 0.25
    x = torch.full((rows, ld), float("nan"), device="cuda", dtype=torch.bfloat16)  # what the pitch's tail holds is nobody's
    x[:, :cols] = torch.randn(rows, cols, generator=gen, device="cuda").bfloat16()
    xd = x[:, :cols].double() * 0.5
    if causal:
        q = torch.arange(rows, device="cuda") % 10
        xd = xd.masked_fill(torch.arange(cols, device="cuda")[None] > q[:, None], float("-inf"))
    ref = torch.softmax(xd, -1)
    keep = K.dropout(torch.ones(rows, cols, device="cuda"), p, salt, seed_tensor=seed)  # the flat mask, scaled
    y, yd, again = torch.empty_like(x), torch.empty_like(x), torch.empty_like(x)
    K.softmax_dropout_fwd(x, y, yd, p, salt, seed, scale=0.5, causal_q=10 if causal else 0, cols=cols)
    _near(y[:, :cols], ref)
    _near(yd[:, :cols], ref * keep)
    assert not y[:, cols:].any() and not yd[:, cols:].any()
    K.dropout_rows(y, again, cols, p, salt, seed)
    _near(again[:, :cols], y[:, :cols].double() * keep)
    dy = torch.full_like(x, float("nan"))
    dy[:, :cols] = torch.randn(rows, cols, generator=gen, device="cuda").bfloat16()
    dx = torch.empty_like(x)
    K.softmax_dropout_bwd(dy, y, dx, p, salt, seed, scale=0.5, cols=cols)
    g, yr = dy[:, :cols].double() * keep, y[:, :cols].double()
    want = 0.5 * yr * (g - (g * yr).sum(-1, keepdim=True))
    # the row sum is one of fp32: its error, up to cols ulps of the sum of magnitudes, times y
    slack = 0.5 * yr * (g * yr).abs().sum(-1, keepdim=True) * cols * 2.0 ** -24
    assert ((dx[:, :cols].double() - want).abs() <= REL * want.abs() + slack + 1e-9).all()


def test_attention_core_with_odd_key_counts():
    """Unfused attention at a key count whose score rows need a pitch, against the fused kernels; dropped probabilities kept and
    formed again."""
    from flexflow_train_b200 import _ffcore as core
    from flexflow_train_b200.runtime.executor import ExecConfig, Executable, OptimizerConfig

    def run(fused, drop, keep):
        cfg = {"batch_size": 2, "sequence_length": 43, "num_heads": 2, "dim_feedforward": 64, "num_features": 128, "num_encoder_layers": 1,
               "num_decoder_layers": 1, "vocab_size": 64, "dropout": drop}
        g = core.build_model("transformer", cfg)
        ex = Executable(g, ExecConfig(seed=3, fused_attention=fused, keep_dropped_probs=keep, optimizer=OptimizerConfig(kind="sgd", lr=0.1)))
        gen = torch.Generator(device="cuda").manual_seed(0)
        ins = {n["name"]: torch.randn(list(n["outputs"][0][1].sizes), generator=gen, device="cuda") for n in g.nodes() if n["type"] == "INPUT"}
        labels = torch.randint(0, 64, (86,), generator=gen, device="cuda", dtype=torch.int32)
        ex.train_step(ins, labels)
        return ex.grads.float().clone()

    a, b = run(False, 0.0, True), run(True, 0.0, True)
    assert (a - b).norm() / b.norm() < 3e-2  # bf16 scores and probabilities against fp32 ones
    a, b = run(False, 0.3, True), run(False, 0.3, False)  # kept and regenerated dropped probabilities: one rounding apart
    assert (a - b).norm() / b.norm() < 1e-2

"""Short kernels launched ahead of each other's end, on buffers whose values change every time."""
import pytest
import torch

pytestmark = pytest.mark.gpu

from flexflow_train_b200.ops import kernels as K  # noqa: E402


@pytest.mark.parametrize("rows,cols", [(64, 256), (2048, 512)])  # kernels of a microsecond or two; of several blocks per SM
@pytest.mark.parametrize("graph", [False, True])
def test_producers_and_consumers_on_one_buffer(rows, cols, graph):
    """Each kernel reads what the one before it wrote, in memory that the iteration before had other values in: launched back to
    back they give, bit for bit, what they give with the device idle between any two."""
    gen = torch.Generator(device="cuda").manual_seed(rows)
    steps = 40
    src = torch.randn(steps, rows, cols, generator=gen, device="cuda")
    x, y, z = (torch.empty(rows, cols, device="cuda", dtype=torch.bfloat16) for _ in range(3))
    t = torch.empty(cols, rows, device="cuda", dtype=torch.bfloat16)
    g, w = torch.empty(cols, device="cuda", dtype=torch.bfloat16), torch.empty(cols, cols, device="cuda", dtype=torch.bfloat16)
    mean, rstd = torch.empty(rows, device="cuda"), torch.empty(rows, device="cuda")
    m, v, master = (torch.zeros(cols, device="cuda") for _ in range(3))
    scratch = torch.empty(max(K.layernorm_bwd_scratch(rows, cols), K.bias_act_bwd_scratch(rows, cols)), device="cuda")

    def run(pause):
        for b in (x, y, z, t, g, w, mean, rstd, m, v, master):
            b.zero_()
        out = []
        for i in range(steps):
            for launch in (lambda: K.cast(src[i], x), lambda: K.cast(src[i, 0], g), lambda: K.cast(src[i].view(-1)[:w.numel()].view_as(w), w)
                           if w.numel() <= src[i].numel() else w.fill_(0.25 / (i + 1)),
                           lambda: K.layernorm_fwd(x, g, g, 1e-5, out=y, mean=mean, rstd=rstd), lambda: K.softmax_fwd(y, out=z),
                           lambda: K.matmul_nt(z, w, out=y), lambda: K.softmax_bwd(y, z, dx=y),
                           lambda: K.layernorm_bwd(y, x, g, mean, rstd, z, g, None, scratch, accumulate_dx=True),
                           lambda: K.transpose2d(z, out=t), lambda: K.bias_act_bwd(z, x, z, g, scratch, "relu", accumulate=True),
                           lambda: K.adam_update(master, m, v, g, None, 1e-2, 0.9, 0.99, 1e-8), lambda: K.axpby(t.view_as(z), z, 0.5, 0.5)):
                launch()
                if pause:
                    torch.cuda.synchronize()
            out += [b.clone() for b in (y, z, g, master)]
        return out

    want = run(True)
    if graph:
        run(False)
        cg = torch.cuda.CUDAGraph()
        with torch.cuda.graph(cg):
            got = run(False)
        cg.replay()
        cg.replay()
    else:
        got = run(False)
    torch.cuda.synchronize()
    bad = [i for i, (a, b) in enumerate(zip(got, want)) if not torch.equal(a.view(torch.uint8), b.view(torch.uint8))]
    assert not bad, bad[:8]

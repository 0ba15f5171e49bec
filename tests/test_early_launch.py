"""Rules of early launches (programmatic dependent launch) that no GPU run could show without a race or a wait that hangs, read
from the kernels' sources."""
import glob
import os
import re

import flexflow_train_b200

SRC = os.path.join(os.path.dirname(flexflow_train_b200.__file__), "csrc", "kernels")


def _sources():
    for path in sorted(glob.glob(os.path.join(SRC, "*.cu")) + glob.glob(os.path.join(SRC, "*.cuh"))):
        text = re.sub(r"/\*.*?\*/", "", open(path).read(), flags=re.S)
        yield os.path.basename(path), re.sub(r"//[^\n]*", "", text)


def _closing(text, at, pair):
    """Index of the bracket that closes the one at `at`."""
    depth = 0
    for i in range(at, len(text)):
        depth += (text[i] == pair[0]) - (text[i] == pair[1])
        if depth == 0:
            return i
    raise AssertionError("unbalanced brackets")


def _kernels():
    """{name: (file, parameters, body)} of every kernel."""
    out = {}
    for name, text in _sources():
        for m in re.finditer(r"__global__", text):
            head = re.compile(r"(?:__launch_bounds__\s*\([^{]*?\)\s*)?(\w+)\s*\(").search(text, text.index("void", m.end()) + 4)
            stop = _closing(text, head.end() - 1, "()")
            brace = text.index("{", stop)
            out[head.group(1)] = (name, text[head.end():stop], text[brace:_closing(text, brace, "{}") + 1])
    return out


KERNELS = _kernels()


def test_every_early_launched_kernel_waits_for_its_predecessor():
    launched = set()
    for _, text in _sources():
        launched |= set(re.findall(r"ffk_launch\(\s*(?:vec::)?(\w+)", text))
        launched |= set(re.findall(r"auto kern = (\w+)", text))
    launched -= {"kern", "void"}
    assert len(launched) > 80 and not launched - set(KERNELS), launched - set(KERNELS)
    late = [k for k in sorted(launched) if not re.search(r"\bpdl_(entry|wait)\s*\(", KERNELS[k][2])]
    assert not late, late


def test_kernels_that_wait_for_peers_do_not_release_their_successor():
    body = KERNELS["gemm_sm100_kernel"][2]
    assert "pdl_entry" not in body
    releases = re.findall(r"if \(!\(([^;]*)\)\) pdl_release\(\);", body)
    assert len(releases) == body.count("pdl_release") == 1
    assert set(re.findall(r"p\.(\w+)", releases[0])) == {"scatter_rows", "gate_flags", "push_src"}
    for name, text in _sources():
        if name == "comm_kernels.cu":
            assert "pdl_" not in text and "ffk_launch" not in text


def test_early_launched_kernels_take_no_input_for_constant():
    """A __restrict__ pointer to const may be read through the non-coherent path, or ahead of the wait, although the
    predecessor still writes there."""
    bad = {k: p for k, (f, p, _) in KERNELS.items() if f != "comm_kernels.cu" for p in re.findall(r"const [\w ]+\*\s*__restrict__ \w+", p)}
    assert not bad, bad
    helpers = [(n, m) for n, text in _sources() if n != "comm_kernels.cu" for m in re.findall(r"const [\w ]+\*\s*__restrict__ \w+", text)]
    assert not helpers, helpers

"""The time limit of a barrier wait is for the kernel's own arrivals.  Under programmatic serialization a kernel may be placed long
before the kernel ahead of it has ended, so every role waits for that one first."""
import os
import re

import pytest
import torch

import portdnn_b200 as pd
from gpu_util import assert_no_device_error

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "portdnn_b200", "csrc")


def _roles():
    """(line, text) of every role of the tensor-core kernels, from its heading to the next."""
    text = open(os.path.join(CSRC, "tc_gemm.cu")).read()
    heads = [m for m in re.finditer(r"^ +// -{20,} (.*?) -{5,}$", text, re.M)]
    ends = [m.start() for m in heads[1:]] + [text.index("// Host side: tensor maps and launch plans")]
    return [(m.group(1), re.sub(r"//[^\n]*", "", text[m.end():end])) for m, end in zip(heads, ends)]


def test_every_role_waits_for_the_preceding_kernel_first():
    roles = [(name, body) for name, body in _roles() if "mbar_wait(" in body]
    assert len(roles) == 4 + 3 + 3 + 3  # persistent, its two pair forms, cluster
    for name, body in roles:
        whole = re.sub(r"if \(grp == 0\) (\{[^{}]*\}|[^;{}]*;)", "", body)  # (what all warps of a role do)
        first = whole.find("grid_dependency_wait();")
        assert 0 <= first < whole.index("mbar_wait("), name


@pytest.mark.gpu
def test_a_long_predecessor_is_no_lost_arrival():
    """A kernel of more than the limit of one second on one SM, and the kernels that are placed on the others meanwhile."""
    pixels = 1000

    def pool(rows):
        return pd.pool_params(1, rows, pixels, 1, rows, 1, False)

    def time(rows):
        q = pool(rows)
        q.window_cols, q.stride_cols, q.out_cols = pixels, 1, 1
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        x = torch.zeros(rows * pixels, device="cuda")
        a.record()
        pd.pooling(pd.POOL_MAX, 0, x, q)
        b.record()
        b.synchronize()
        return a.elapsed_time(b) / 1000, x, q

    time(100)
    per_row = time(1000)[0] / 1000
    rows = int(1.5 / per_row)
    g = torch.Generator(device="cuda").manual_seed(2)

    def layer(n, h, c, k, win, dtype, **args):
        p = pd.conv_params(n, h, h, c, k, win, 1)
        x = torch.randn(n * h * h * c, device="cuda", generator=g).to(dtype)
        w = (torch.randn(win * win * c * k, device="cuda", generator=g) * 0.05).to(dtype)
        return lambda: pd.conv2d(pd.FORWARD, x, w, p, **args)

    layers = [layer(64, 28, 256, 128, 1, torch.half), layer(8, 28, 64, 96, 3, torch.float32), layer(1, 14, 512, 256, 1, torch.half, any_order=True)]
    for run in layers:
        want = run()
        seconds, x, q = time(rows)
        assert seconds > 1.1
        pd.pooling(pd.POOL_MAX, 0, x, q)
        got = run()
        assert torch.equal(got, want)
        assert_no_device_error()

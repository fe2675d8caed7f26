"""constant_filter speaks of the caller's filter.  An NCHW layer reads a copy of it that the launch right ahead of the layer writes,
so the layer may not request its filter before that launch has ended."""
import os
import re

import pytest
import torch

import portdnn_b200 as pd

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "portdnn_b200", "csrc")


def test_the_flag_stays_behind():
    """Read in the source: the layer between the transposes gets copies of the caller's structures with the flag cleared."""
    text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, "c_api.cu")).read())
    branch = text[text.index("p->input_format == 1) {\n"):]
    branch = branch[:branch.index("\n  }\n")]
    cleared = re.search(r"(\w+)\.constant_filter = (\w+)\.constant_filter = 0;", branch)
    assert cleared, "constant_filter reaches the layer"
    call = branch[branch.index("dispatch_conv("):]
    passed = re.findall(r"&(\w+)", call[:call.index(");")])
    assert set(cleared.groups()) <= set(passed) and not re.search(r"[(,] (epi|fusion),", call)


# filters streamed through the ring by persistent CTAs, by small CTAs, held in shared memory
@pytest.mark.gpu
@pytest.mark.parametrize("n,h,c,k,win", [(40, 28, 256, 512, 3), (3, 14, 512, 128, 1), (64, 28, 64, 64, 1)])
def test_each_call_reads_its_own_filter(n, h, c, k, win):
    p, q = pd.conv_params(n, h, h, c, k, win, 1), pd.conv_params(n, h, h, c, k, win, 1)
    q.input_format, q.filter_format = 1, 1
    g = torch.Generator(device="cuda").manual_seed(c)
    x, dy = torch.randn(n, h, h, c, device="cuda", generator=g).half(), torch.randn(n, h, h, k, device="cuda", generator=g).half()
    nchw = lambda t: t.permute(0, 3, 1, 2).contiguous().reshape(-1)  # noqa: E731
    xs, ds = nchw(x), nchw(dy)
    for i in range(4):  # another filter each time, in scratch that holds the copy of the one before
        w = (torch.randn(win, win, c, k, device="cuda", generator=g) * 0.05).half()
        ws = w.permute(3, 2, 0, 1).contiguous().reshape(-1)
        y = pd.conv2d(pd.FORWARD, x.reshape(-1), w.reshape(-1), p).view(n, h, h, k)
        dx = pd.conv2d(pd.INPUT_BACKPROP, dy.reshape(-1), w.reshape(-1), p).view(n, h, h, c)
        args = {"algorithm": pd.ALGO_DIRECT, "constant_filter": True}
        assert torch.equal(pd.conv2d(pd.FORWARD, xs, ws, q, **args), nchw(y))
        assert torch.equal(pd.conv2d(pd.INPUT_BACKPROP, ds, ws, q, **args), nchw(dx))

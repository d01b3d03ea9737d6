"""Kernels that are placed before their predecessor has ended: what they read, they read by ordinary loads behind the wait."""
import glob
import os
import re

import pytest

from tsplit_b200 import ndarray
from tsplit_b200.ops import _gpu as G

KERNELS = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "tsplit_b200", "csrc", "kernels")


def _code(path):
    text = open(path).read()
    return re.sub(r"/\*.*?\*/", "", re.sub(r"//[^\n]*", "", text), flags=re.S)


def test_no_read_only_loads():
    """``ld.global.nc`` wants data that is constant for the whole life of a kernel, which begins before its inputs are
    written: no ``__ldg``, no such PTX, no ``const`` pointer with ``__restrict__`` (nvcc turns its loads into it)."""
    files = glob.glob(os.path.join(KERNELS, "*.cu")) + glob.glob(os.path.join(KERNELS, "*.cuh"))
    assert len(files) >= 10
    for path in files:
        code = _code(path)
        for what in (r"\b__ldg\b", r"ld\.global[a-z.0-9:]*\.nc", r"const\s+\w+(\s+const)?\s*\*\s*(const\s*)?__restrict__",
                     r"\w+\s+const\s*\*\s*(const\s*)?__restrict__"):
            assert not re.search(what, code), (os.path.basename(path), what)


@pytest.mark.gpu
@pytest.mark.parametrize("blocks", [1, 31, 32, 33])
def test_small_writers_and_their_readers_in_a_captured_chain(blocks):
    """One buffer, written by a kernel of few blocks (which lets the next be placed at once), read by the next one,
    and written again: the sums of what was read are those of running the kernels one at a time."""
    import torch
    from tsplit_b200.runtime import cudagraph
    from tsplit_b200.stream import create_stream_handle
    ctx = ndarray.gpu(0)
    st = create_stream_handle(ctx)
    n = 2048 * blocks
    arr = lambda t: ndarray.from_tensor(t, ctx)
    x, buf, acc = (torch.zeros(n, device="cuda") for _ in range(3))
    ids, rows, table = torch.zeros(64, device="cuda"), torch.zeros(64, 32, device="cuda"), torch.ones(4, 32, device="cuda")
    bias, wide, shifted = torch.zeros(64, device="cuda"), torch.zeros(n // 64, 64, device="cuda"), torch.zeros(n // 64, 64, device="cuda")
    sums = torch.zeros(64, device="cuda")
    torch.cuda.synchronize()

    def step():
        for k in range(8):
            G.unary(G.UN_ADDC, arr(x), arr(x), st, alpha=1.0)                     # x counts the kernels
            G.unary(G.UN_MULC, arr(x), arr(buf), st, alpha=float(2 * k + 1))      # writes
            G.binary(G.BIN_ADD, arr(acc), arr(buf), arr(acc), st)                 # reads at once
            G.fill(arr(ids), float(k % 4), st)
            G.embedding(arr(table), arr(ids), arr(rows), st)                      # ids written just before
            G.fill(arr(bias), float(k), st)
            G.add_broadcast(arr(wide), arr(bias), [0, 1], arr(shifted), st)       # the row written just before
            G.reduce_sum(shifted.data_ptr(), [n // 64, 64], [64, 1], [0], arr(sums), st)
            G.binary(G.BIN_MUL, arr(table), arr(table), arr(table), st)
    step()
    st.sync()
    graph = cudagraph.capture(st, step)
    replays = 200
    for _ in range(replays):
        graph.launch(st)
    st.sync()
    want, count = 0.0, 0
    for _ in range(replays + 1):
        for k in range(8):
            count += 1
            want += (count * (2 * k + 1))
    assert want < 2 ** 24                                   # whole numbers below 2^24: every sum is exact
    assert torch.all(x == count) and torch.all(acc == want)
    assert torch.all(rows == 1) and torch.all(shifted == 7) and torch.all(sums == 7 * (n // 64))

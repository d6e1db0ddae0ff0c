"""Launches prepared while the kernel before them runs keep the stream's order:
the library's kernels between other kernels of one stream, on a stream of its
own, on the default stream and in a captured graph, against the same calls with
a synchronisation behind each."""
import numpy as np
import pytest

from conftest import rand_fe

pytestmark = pytest.mark.gpu

P = (1 << 61) - 1


def chain(ctx, gbz, torch, x, logn, steps, wait):
    for k in range(steps):
        x.copy_(torch.flip(x, (0,)))
        wait()
        ctx.check(gbz.lib.gbz_fft(ctx.h, x.data_ptr(), logn, k & 1, gbz.MEM_DEVICE))
        wait()


@pytest.mark.parametrize("how", ["own", "default", "graph"])
@pytest.mark.parametrize("logn", [3, 10, 13, 16, 21])
def test_order(gbz, how, logn):
    torch = pytest.importorskip("torch")
    x0 = torch.from_numpy(rand_fe(np.random.default_rng(logn), 1 << logn).view(np.int64)).cuda()
    c = gbz.Context(0)
    ref, x = x0.clone(), x0.clone()
    s = torch.cuda.Stream() if how != "default" else torch.cuda.default_stream()
    c.set_stream(s.cuda_stream)
    torch.cuda.synchronize()
    with torch.cuda.stream(s):
        chain(c, gbz, torch, ref, logn, 9, torch.cuda.synchronize)  # the tables are built here
        if how == "graph":
            g = torch.cuda.CUDAGraph()
            with torch.cuda.graph(g, stream=s):
                chain(c, gbz, torch, x, logn, 9, lambda: None)
            g.replay()
        else:
            chain(c, gbz, torch, x, logn, 9, lambda: None)
    torch.cuda.synchronize()
    assert torch.equal(x, ref)
    c.set_stream(torch.cuda.Stream().cuda_stream)
    c.close()

"""Sorts, whose passes are launched while the ones before them run, on a caller's stream beside its own work and
inside a caller's capture, replayed on other keys: every size class, low digits set by the high ones and not."""
import ctypes

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("what", ["set", "few", "full"])
@pytest.mark.parametrize("n", [3000, 300001, (2 << 20) + 77])
def test_sort_on_a_stream_and_captured(n, what):
    torch = pytest.importorskip("torch")
    from fluidloom_gb300 import Context
    stream = torch.cuda.Stream()
    ctx = Context(0)
    ctx.set_stream(stream.cuda_stream)
    k = torch.empty(n, dtype=torch.int64, device="cuda")
    i = torch.empty(n, dtype=torch.int32, device="cuda")

    def keys(seed):
        g = torch.Generator(device="cuda")
        g.manual_seed(seed)
        top = torch.randint(0, 1 << (20 if what == "few" else 30), (n,), device="cuda", generator=g)
        low = torch.randint(0, 1 << 33, (n if what == "full" else 11,), device="cuda", generator=g)
        if what != "full":
            low = low[top % 11 if what == "set" else torch.randint(0, 11, (n,), device="cuda", generator=g)]
        torch.cuda.synchronize()
        return (top << 33) | low

    def sort():
        ctx.call("fl_sort_pairs_u64_u32", ctypes.c_void_p(k.data_ptr()), ctypes.c_void_p(i.data_ptr()), ctypes.c_size_t(n), 0, 63)

    def check(a, got_k, got_i):
        want, order = torch.sort(a, stable=True)
        assert torch.equal(got_k, want) and torch.equal(got_i, order.int())

    for seed in (1, 2):
        a = keys(seed)
        with torch.cuda.stream(stream):  # filled before and copied after the sort, no wait between
            k.copy_(a)
            torch.arange(n, dtype=torch.int32, device="cuda", out=i)
            sort()
            got = k.clone(), i.clone()
            k.zero_()
        torch.cuda.synchronize()
        check(a, *got)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        sort()
    for seed in (3, 4):
        a = keys(seed)
        k.copy_(a)
        torch.arange(n, dtype=torch.int32, device="cuda", out=i)
        torch.cuda.synchronize()
        graph.replay()
        torch.cuda.synchronize()
        check(a, k, i)
    ctx.close()

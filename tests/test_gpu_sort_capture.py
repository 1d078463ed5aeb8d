"""Sorts recorded into a CUDA graph: behind a copy, a memset and a kernel, and on
a stream that joined another one; replayed with other keys, other counts and
another schedule. Every replay equals a stable sort."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [300, 3000, 50000, 300000, 2200000])
@pytest.mark.parametrize("before", ["copy", "memset", "kernel", "join"])
def test_captured_sorts_replay(native, n, before):
    import torch

    from astro_gb300.radix_sort import RadixSort

    gen = torch.Generator(device="cuda").manual_seed(n)
    source = torch.empty(n, dtype=torch.int64, device="cuda")
    keys, keys_out = torch.empty_like(source), torch.empty_like(source)
    index = torch.arange(n, dtype=torch.int32, device="cuda")
    index_out = torch.empty_like(index)
    count = torch.tensor([n], dtype=torch.int32, device="cuda")
    cleared = torch.empty(1 << 20, dtype=torch.uint8, device="cuda")
    sorter = RadixSort(n, 63)
    sorter.sort(source.random_(generator=gen), index, keys_out, index_out, n, count)  # set-up before the capture
    other = torch.cuda.Stream()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        stream = torch.cuda.current_stream()
        if before == "join":
            other.wait_stream(stream)
            with torch.cuda.stream(other):
                keys.copy_(source)
                cleared.zero_()
            index_out.fill_(-1)
            stream.wait_stream(other)
        else:
            keys.copy_(source)
            if before == "memset":
                cleared.zero_()
            elif before == "kernel":
                keys.bitwise_and_((1 << 63) - 1)
        sorter.sort(keys, index, keys_out, index_out, n, count, stream=stream.cuda_stream)
        keys.add_(1)  # behind the sort: must not reach its input
    for k in range(4):
        source.random_(generator=gen)
        if k == 1:
            source.bitwise_and_(0xFFFFFF)  # other digits
        if k == 2:
            source[: n // 2] = source[0]  # a run too long for the top digits
        m = n if k != 3 else n - n // 3
        count.fill_(m)
        graph.replay()
        torch.cuda.synchronize()
        want, order = torch.sort(source[:m], stable=True)
        assert torch.equal(keys_out[:m], want)
        assert torch.equal(index_out[:m].long(), order)

"""Time of one launch on the device: launches captured into a graph, the best of several replays."""


def us(torch, launch, n=20):
    """`launch(stream)` returns 0; microseconds each of `n` back to back."""
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        assert launch(side.cuda_stream) == 0
        side.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=side):
            for _ in range(n):
                assert launch(side.cuda_stream) == 0
        best = float("inf")
        for _ in range(8):
            begin, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            begin.record(side)
            graph.replay()
            end.record(side)
            side.synchronize()
            best = min(best, begin.elapsed_time(end) * 1e3 / n)
    return best

"""Launches that add up parts through scratch of the library (attention with few query rows, array reductions) on many
streams, in graphs and on threads at the same time: every launch gives what it gives alone."""
import ctypes as C
import threading

import pytest

pytestmark = pytest.mark.gpu


class Work:
    """A decode step and a column sum on inputs of its own, with the results of a run on its own."""

    def __init__(self, cuda, seed):
        import torch
        g = torch.Generator(device="cuda").manual_seed(seed)
        r = lambda *s: torch.randn(*s, device="cuda", generator=g)
        self.cuda, self.q = cuda, r(1, 8, 1, 64).half()
        self.k, self.v = r(1, 2, 3000, 64).half(), r(1, 2, 3000, 64).half()
        self.a = r(3000, 256)
        self.want = self.run()

    def run(self):
        T = self.cuda.tiled
        o = self.cuda.fmha.cutile_fmha(self.q, self.k, self.v, causal=True, input_pos=2999, query_group_size=4)
        return o, T.tsum(T.Tiled(self.a), dims=2), T.tsum(T.Tiled(self.a))

    def check(self, got):
        import torch
        for a, b in zip(got, self.want):
            assert torch.equal(a, b)


@pytest.fixture
def streams():
    """Distinct streams (torch hands out a pool of 32)."""
    import torch
    rt = torch.cuda.cudart()
    made = []

    def make(n):
        for _ in range(n):
            h = C.c_void_p()
            assert int(rt.cudaStreamCreate(C.addressof(h))) == 0
            made.append(h.value)
        return [torch.cuda.ExternalStream(h) for h in made[-n:]]
    yield make
    torch.cuda.synchronize()
    for h in made:
        rt.cudaStreamDestroy(h)


def test_more_streams_than_slots(cuda, streams):
    import torch
    work = [Work(cuda, s) for s in range(6)]
    torch.cuda.synchronize()
    many = streams(150)
    for _ in range(3):
        got = []
        for i, st in enumerate(many):
            with torch.cuda.stream(st):
                got.append((i % 6, work[i % 6].run()))
        torch.cuda.synchronize()
        for i, g in got:
            work[i].check(g)
    cuda.check_device_status(0)


def test_captures_survive_a_change_of_owners(cuda, streams):
    """Eager launches on more streams than there are slots, while a graph is being captured."""
    import torch
    work = [Work(cuda, s) for s in range(2)]
    side, *many = streams(130)
    for st in many:  # every slot has an owner
        with torch.cuda.stream(st):
            work[1].run()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    got = []

    def other():
        with torch.cuda.stream(many[0]):
            got.append(work[1].run())
        for st in many[:40]:
            with torch.cuda.stream(st):
                got.append(work[1].run())
    with torch.cuda.graph(graph, stream=side, capture_error_mode="thread_local"):
        out = work[0].run()
        t = threading.Thread(target=other)
        t.start()
        t.join()
        more = work[0].run()
    graph.replay()
    torch.cuda.synchronize()
    work[0].check(out)
    work[0].check(more)
    assert len(got) == 41
    for g in got:
        work[1].check(g)


def test_graphs_of_one_stream_replayed_side_by_side(cuda, streams):
    import torch
    work = [Work(cuda, s) for s in range(4)]
    side, a, b, c = streams(4)
    graphs, outs = [], []
    torch.cuda.synchronize()
    for w in work[:3]:
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=side):
            outs.append(w.run())
        graphs.append(graph)
    for _ in range(40):
        for o in outs:
            for t in o:
                t.zero_()
        torch.cuda.synchronize()
        for st, graph in zip((a, b, c), graphs):
            with torch.cuda.stream(st):
                for _ in range(5):
                    graph.replay()
        with torch.cuda.stream(side):  # eager work on the stream of the captures
            eager = [work[3].run() for _ in range(5)]
        torch.cuda.synchronize()
        for w, o in zip(work, outs):
            w.check(o)
        for e in eager:
            work[3].check(e)
    cuda.check_device_status(0)


def test_a_capture_with_two_branches(cuda, streams):
    import torch
    work = [Work(cuda, s) for s in range(2)]
    side, fork = streams(2)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=side):
        fork.wait_stream(side)
        with torch.cuda.stream(fork):
            second = work[1].run()
        first = work[0].run()
        side.wait_stream(fork)
    for _ in range(50):
        graph.replay()
    torch.cuda.synchronize()
    work[0].check(first)
    work[1].check(second)


def test_graphs_give_their_scratch_back(cuda, streams):
    import torch
    w = Work(cuda, 0)
    side, = streams(1)
    torch.cuda.synchronize()

    def capture():
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=side):
            out = w.run()
        graph.replay()
        torch.cuda.synchronize()
        w.check(out)
    for _ in range(4):
        capture()
    torch.cuda.empty_cache()
    free = torch.cuda.mem_get_info()[0]
    for _ in range(120):
        capture()
    torch.cuda.empty_cache()
    assert free - torch.cuda.mem_get_info()[0] < 64 << 20  # 120 slots of 1.25 MB would be 150


def test_threads(cuda, streams):
    import torch
    work = [Work(cuda, s) for s in range(6)]
    torch.cuda.synchronize()
    many, wrong = streams(6), []

    def loop(w, st):
        with torch.cuda.stream(st):
            for _ in range(60):
                got = w.run()
                st.synchronize()
                try:
                    w.check(got)
                except AssertionError as e:
                    wrong.append(e)
    threads = [threading.Thread(target=loop, args=p) for p in zip(work, many)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong

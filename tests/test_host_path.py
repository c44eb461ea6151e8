"""The native call path of the package (csrc/host.cpp): expression nodes without a GPU, and on a GPU that calls it takes
itself and calls it leaves to the Python checks give the same results."""
import numpy as np
import pytest


def test_expression_nodes():
    import torch
    from cutile_b200 import tiled as T
    e = T.Expr.wrap(2) + 3
    assert e.node[0] == "add" and e.node[1].node == ("const", 2.0) and isinstance(e, T.Expr)
    assert (2.0 * e).node[0] == "mul" and (2.0 * e).node[2] is e
    assert [(-e).node[0], abs(e).node[0], (e ** 2).node[0], T.tanh(e).node[0], T.tmax(e, 1).node[0]] == \
        ["neg", "abs", "pow", "tanh", "max"]
    with pytest.raises(TypeError):
        2 ** e
    with pytest.raises(TypeError):
        e + range(3)
    with pytest.raises(ValueError, match="device memory"):
        T.Tiled(torch.ones(3))
    for _ in range(20000):  # a tree this deep is released without recursion
        e = e + 1.0
    del e


def test_function_forms_take_keywords():
    from cutile_b200 import tiled as T
    e = T.Expr.wrap(2.0)
    assert T.sin(x=e).node == ("sin", e) and T.abs2(x=e).node == ("abs2", e)
    assert T.tmax(a=e, b=1).node[:2] == ("max", e) and T.tmin(1, b=e).node[2] is e


def test_nodes_are_ordinary_objects():
    """Copies, pickles, weak references and attributes of their own, also in subclasses."""
    import copy
    import gc
    import pickle
    import weakref

    from cutile_b200 import tiled as T
    e = T.Expr.wrap(2.0) * 3.0 + T.exp(T.Expr.wrap(0.5))
    for c in (copy.copy(e), copy.deepcopy(e), pickle.loads(pickle.dumps(e))):
        assert type(c) is T.Expr and c.node[0] == "add" and c.node[1].node[0] == "mul" and c.node[2].node[1].node == ("const", 0.5)
    assert copy.copy(e).node[1] is e.node[1]
    e.label = "sum"
    assert copy.copy(e).label == "sum" and e.__dict__ == {"label": "sum"}
    r = weakref.ref(e)
    assert r() is e
    e.label = e  # a cycle
    del e, c
    gc.collect()
    assert r() is None

    class Named(T.Expr):
        def __init__(self, name, *node):
            super().__init__(*node)
            self.name = name
    n = Named("two", "const", 2.0)
    c = copy.copy(n)
    assert type(c) is Named and c.name == "two" and c.node == ("const", 2.0)
    assert n.name == "two" and (n + 1).node[1] is n and weakref.ref(n)() is n


@pytest.mark.gpu
@pytest.mark.parametrize("m,n", [(1, 4), (64, 1000), (33, 4096)])
def test_native_and_checked_calls_agree(cuda, m, n):
    import torch
    g = torch.Generator(device="cuda").manual_seed(1)
    x = torch.randn(m, n, device="cuda", generator=g)
    outs = []
    for hints in ({}, {"occupancy": 2}):  # launch keywords take the Python path
        o = torch.full_like(x, float("nan"))
        assert cuda.softmax.softmax_chunked_kernel(o, x, n, 1024, **hints) is o
        a = torch.full_like(x, float("nan"))
        cuda.tiled.assign(a, cuda.tiled.Tiled(x) * 2.0 + cuda.tiled.tanh(cuda.tiled.Tiled(x[:1].contiguous())), **hints)
        s = cuda.tiled.tsum(cuda.tiled.Tiled(x), dims=1, **hints)
        v = cuda.vadd.vec_add_kernel_2d(x, o, torch.empty_like(x), 32, 32, **hints)
        outs.append([t.cpu().numpy() for t in (o, a, s, v)])
    for p, q in zip(*outs):
        assert p.shape == q.shape and np.array_equal(p, q)


@pytest.mark.gpu
def test_native_path_follows_the_current_stream(cuda):
    import torch
    x = torch.randn(4096, 4096, device="cuda")
    want = torch.softmax(x, 1)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        y = x * 1.0
        o = torch.empty_like(y)
        cuda.softmax.softmax_tma_kernel(o, y, 4096)
    side.synchronize()
    assert (o - want).abs().max().item() < 1e-6


@pytest.mark.gpu
def test_tensors_without_data_raise(cuda):
    """Fake tensors and those that vmap passes have no address: an ordinary exception, and the interpreter goes on."""
    import threading

    import torch
    from torch._subclasses.fake_tensor import FakeTensorMode
    T = cuda.tiled
    x = torch.randn(3, 8, 64, device="cuda")
    o = torch.empty(8, 64, device="cuda")
    calls = [lambda t: cuda.softmax.softmax_tma_kernel(o, t, 64), lambda t: T.tsum(T.Tiled(t)),
             lambda t: T.assign(o, T.Tiled(t) + 1.0), lambda t: cuda.vadd.vec_add_kernel_2d(t, t, o, 32, 32),
             lambda t: cuda.transpose.transpose_kernel(t, torch.empty(64, 8, device="cuda"), 32, 32),
             lambda t: cuda.fmha.cutile_fmha(*3 * (t.half().reshape(1, 1, 8, 64),))]
    fake = FakeTensorMode().from_tensor(x[0].clone())
    for call in calls:
        with pytest.raises(RuntimeError):
            call(fake)
        with pytest.raises(RuntimeError):
            torch.vmap(call)(x)
    ran = []
    t = threading.Thread(target=lambda: ran.append(call(x[0])))
    t.start()
    t.join()
    assert len(ran) == 1 and ran[0].shape == (1, 1, 8, 64)


@pytest.mark.gpu
def test_threads_with_different_sizes(cuda):
    """Calls of one kernel that need different amounts of shared memory, from several threads at once."""
    import threading

    import torch
    g = torch.Generator(device="cuda").manual_seed(2)
    r = lambda *s: torch.randn(*s, device="cuda", generator=g)
    T, jobs = cuda.tiled, []

    def softmax(n):
        x = r(4, n)
        jobs.append(lambda: cuda.softmax.softmax_chunked_kernel(torch.empty_like(x), x, n, 1024))

    def layernorm(n):
        x, w, m = r(8, n), r(n), torch.ones(8, device="cuda")
        e = lambda: torch.empty(8, n, device="cuda")

        def run():
            cuda.layernorm.layer_norm_fwd(x, w, w, e(), torch.empty(8, device="cuda"), torch.empty(8, device="cuda"), 1e-5, 1024)
            cuda.layernorm.layer_norm_bwd_dx_partial_dwdb(e(), x, e(), e(), x, w, m, m, None, 8, 1024)
        jobs.append(run)

    def sums(k):
        a = [T.Tiled(r(64, 1024)) for _ in range(k)]
        jobs.append(lambda: T.materialize(sum(a[1:], a[0] * 2.0)))

    def transform(f):
        x, plan = torch.view_as_complex(r(4, f[0] * f[1] * f[2], 2)), cuda.fft.FftPlan(f, "cuda")
        jobs.append(lambda: plan(x))
    softmax(9000), softmax(26000), softmax(4096), softmax(8192), layernorm(2048), layernorm(1028), layernorm(8192)
    layernorm(8191), layernorm(2047), layernorm(300), layernorm(1023), sums(2), sums(3), transform((16, 16, 16)), transform((32, 16, 16))
    wrong = []

    def loop(job):
        try:
            for _ in range(300):
                job()
        except Exception as e:  # noqa: BLE001
            wrong.append(e)
    threads = [threading.Thread(target=loop, args=(j,)) for j in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert not wrong, wrong[0]

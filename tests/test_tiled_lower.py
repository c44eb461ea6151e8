"""The program that the broadcast kernel runs (ctb_tiled_lower), without a GPU: a numpy machine with the documented meaning of
its words gives the value of the expression evaluated operator by operator in f32, bit for bit: every word is made so that its
result is the operator's own (constants, negation and shared subexpressions included)."""
import ctypes as C

import numpy as np
import pytest

from test_tiled_compile import OPS, postfix, size

F = np.float32
UNARY = {"identity": lambda x: x, "neg": lambda x: -x, "abs": np.abs, "sqrt": np.sqrt, "exp": np.exp, "exp2": np.exp2, "log": np.log,
         "log2": np.log2, "sin": np.sin, "cos": np.cos, "tanh": np.tanh, "inv": lambda x: F(1) / x, "abs2": lambda x: x * x}
BINARY = {"add": np.add, "sub": np.subtract, "mul": np.multiply, "div": np.divide, "max": np.fmax, "min": np.fmin, "pow": np.power}
NAMES = {v: k for k, v in OPS.items()}
COLD = ["sub", "div", "max", "min", "pow"]
TEMPS, MAX_OPS, MAX_WORDS = 4, 32, 48


def lower(tree, n_inputs, consts):
    from cutile_b200 import _lib as L
    prog = postfix(tree, [])
    words, pq, n, t = (C.c_uint32 * MAX_WORDS)(), (C.c_float * (2 * MAX_WORDS))(), C.c_int(-1), C.c_int(-1)
    st = L.lib.ctb_tiled_lower((C.c_int32 * len(prog))(*prog), len(prog) // 2, n_inputs, (C.c_float * max(1, len(consts)))(*consts),
                               len(consts), words, pq, C.byref(n), C.byref(t))
    assert st == 0, L.last_error()
    assert 0 < n.value <= MAX_WORDS and 0 <= t.value <= TEMPS
    return [(words[k], F(pq[2 * k]), F(pq[2 * k + 1])) for k in range(n.value)], t.value


def fma(x, p, q):
    """p x + q rounded once: the product is exact in f64, and rounding an f64 sum of f32 values again to f32 is the same as
    rounding the sum once (53 >= 2 * 24 + 2).  Holds for p = +-1 and for q = -0, the only forms there are."""
    assert abs(p) == 1 or (q == 0 and np.signbit(q)) or np.isnan(p)
    return (np.float64(p) * x.astype(np.float64) + np.float64(q)).astype(F)


def run(words, n_temps, inputs):
    acc, temps = None, {}

    def temp(a):
        assert a < n_temps
        return temps[a]
    for w, p, q in words:
        op, a = w & 0xFF, (w >> 8) & 3
        if op == 0:
            acc = fma(acc, p, q)
        elif op in (1, 2):
            acc = inputs[a] if op == 1 else temp(a)
        elif op in (3, 4, 5, 6):
            x = inputs[a] if op in (3, 5) else temp(a)
            if w & 1 << 11:
                x = fma(x, p, q)
            acc = acc * x if op in (3, 4) else acc - x if w & 1 << 10 else acc + x
        elif op == 7:
            acc = np.full_like(inputs[0], q)
        elif op < 20:
            acc = UNARY[NAMES[OPS["neg"] + op - 8]](acc)
        else:
            s, j = divmod(op - 20, 10)
            x = (lambda: inputs[a], lambda: np.full_like(inputs[0], q), lambda: temp(a))[s]()
            f = BINARY[COLD[j // 2]]
            acc = f(x, acc) if j % 2 else f(acc, x)
        if w & 1 << 12:
            assert op not in (0, 7) and not w & 1 << 11 and not 30 <= op < 40  # p and q are free for it
            acc = fma(acc, p, q)
        if w >> 13:
            assert (w >> 13) - 1 < n_temps
            temps[(w >> 13) - 1] = acc
    return acc


def value(tree, inputs, consts):
    if tree[0] == "in":
        return inputs[tree[1]]
    if tree[0] == "c":
        return np.full_like(inputs[0], F(consts[tree[1]]))
    f = UNARY.get(tree[0]) or BINARY[tree[0]]
    return f(*(value(c, inputs, consts) for c in tree[1:]))


def same(a, b):
    nan = np.isnan(a) & np.isnan(b)
    return bool(np.all(nan | ((a == b) & (np.signbit(a) == np.signbit(b)))))


def check(tree, inputs, consts):
    words, n_temps = lower(tree, len(inputs), consts)
    with np.errstate(all="ignore"):
        got, want = run(words, n_temps, inputs), value(tree, inputs, consts)
    assert got.dtype == want.dtype == F and same(np.broadcast_to(got, want.shape), want), (tree, words)
    return words, n_temps


def random_inputs(g):
    special = np.array([0.0, -0.0, 1.0, -1.0, np.inf, -np.inf, np.nan, 1e-40, -1e-45, 3e38, -3e38], F)
    x = [(g.standard_normal(64) * 10.0 ** g.integers(-3, 4, 64)).astype(F) for _ in range(4)]
    for v in x:
        v[: len(special)] = g.permutation(special)
    return x


def random_tree(g, budget, pool):
    """Subtrees come again with some probability, so that values are shared."""
    if pool and g.random() < 0.25:
        t = pool[int(g.integers(0, len(pool)))]
        if size(t) <= budget:
            return t
    if budget <= 1 or g.random() < 0.1:
        t = ("in", int(g.integers(0, 4))) if g.random() < 0.65 else ("c", int(g.integers(0, 6)))
    elif g.random() < 0.25:
        names = [u for u in UNARY if u not in ("exp2", "log2")]
        t = (names[int(g.integers(0, len(names)))], random_tree(g, budget - 1, pool))
    else:
        names = ["add", "sub", "mul", "add", "sub", "mul", "div", "max", "min", "pow"]
        left = int(g.integers(1, budget - 1)) if budget > 2 else 1
        t = (names[int(g.integers(0, len(names)))], random_tree(g, left, pool), random_tree(g, max(1, budget - 1 - left), pool))
    pool.append(t)
    return t


@pytest.mark.parametrize("seed", range(8))
def test_random_programs(seed):
    g = np.random.default_rng(seed)
    done = temps = 0
    while done < 1000:
        tree = random_tree(g, int(g.integers(1, MAX_OPS + 1)), [])
        if size(tree) > MAX_OPS:
            continue
        consts = [0.5, -0.0, 0.0, 3.0, float(F(g.standard_normal())), float(g.choice([np.inf, 1.0, -1.0, 1e-38]))]
        temps = max(temps, check(tree, random_inputs(g), consts)[1])
        done += 1
    assert temps >= 3


def test_longest_programs():
    """Thirty-two operations of the kinds that need most words and most values at once."""
    g = np.random.default_rng(3)
    inputs, most, temps = random_inputs(g), 0, 0

    def full(depth, leaf):
        return leaf() if depth == 0 else (("sub", "div", "add", "mul")[int(g.integers(0, 4))], full(depth - 1, leaf), full(depth - 1, leaf))
    for _ in range(2000):
        kind = int(g.integers(0, 4))
        leaf = lambda: (("in", int(g.integers(0, 4))), ("mul", ("in", int(g.integers(0, 4))), ("c", 0)), ("sin", ("in", int(g.integers(0, 4)))),
                        ("sub", ("c", 1), ("neg", ("in", 1))))[kind if g.random() < 0.7 else int(g.integers(0, 4))]
        tree = full(int(g.integers(2, 5)), leaf)
        while size(tree) <= MAX_OPS - 2 and g.random() < 0.9:
            tree = ("add", tree, ("in", 2)) if g.random() < 0.5 else ("neg", tree)
        if size(tree) <= MAX_OPS:
            words, n_temps = check(tree, inputs, [1.5, -2.0])
            most, temps = max(most, len(words)), max(temps, n_temps)
    assert most >= 20 and temps == TEMPS


def test_what_the_kernel_is_said_to_run():
    # 0.5 v (1 + tanh(c (v + k v v v))), v = x + b: v in one temporary, seven words
    v = ("add", ("in", 0), ("in", 1))
    cube = ("mul", ("mul", v, v), v)
    tree = ("mul", ("mul", ("c", 0), v), ("add", ("c", 1), ("tanh", ("mul", ("c", 2), ("add", v, ("mul", ("c", 3), cube))))))
    words, n_temps = check(tree, random_inputs(np.random.default_rng(0)), [0.5, 1.0, 0.7978845608, 0.044715])
    assert len(words) == 7 and n_temps == 1
    words, n_temps = check(("add", ("mul", ("c", 0), ("in", 0)), ("c", 1)), random_inputs(np.random.default_rng(1)), [2.0, 1.0])
    assert len(words) == 2 and n_temps == 0


def test_scaled_operand_takes_no_temporary():
    # (x + c) (y + d): y enters as y + d, without a temporary
    tree = ("mul", ("add", ("in", 0), ("c", 0)), ("add", ("in", 1), ("c", 1)))
    words, n_temps = check(tree, random_inputs(np.random.default_rng(2)), [2.0, 1.0])
    assert any(w & 1 << 11 for w, _, _ in words) and n_temps == 0


@pytest.mark.parametrize("prog,frag", [([64, 0], "needs two values"), ([0, 2], "input that was not given"), ([0, 0, 99, 0], "not an operation")])
def test_malformed_programs(prog, frag):
    from cutile_b200 import _lib as L
    words, pq, n = (C.c_uint32 * MAX_WORDS)(), (C.c_float * (2 * MAX_WORDS))(), C.c_int()
    st = L.lib.ctb_tiled_lower((C.c_int32 * len(prog))(*prog), len(prog) // 2, 1, None, 0, words, pq, C.byref(n), C.byref(n))
    assert st == L.BAD_ARG and frag in L.last_error()

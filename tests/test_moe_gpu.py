"""GPU parity of the MoE kernels against the oracle.

Routing (top-k ids, sorted slot ids, expert ids per block) must be bit-exact;
router logits are compared bit for bit with the float32 CPU loop; gate weights
within one f16 ulp (expf differs between CPU and GPU); FFN outputs within a
relative Frobenius error of 2e-3 (f16 operands, f32 accumulation, f16 output).
The reference's own check is norm-wise rtol=1e-2, atol=1e-2 (examples/moe.jl:370-374)."""
import numpy as np
import pytest

from oracle import inputs, ref

pytestmark = pytest.mark.gpu
TOL = 2e-3


def random_routing(T, E, topk, seed):
    """ids and weights drawn the way the reference's prepare() does (examples/moe.jl:323-332)."""
    g = np.random.default_rng(seed)
    ids = np.stack([g.permutation(E)[:topk] + 1 for _ in range(T)], axis=1).astype(np.int64)  # [topk, T]
    raw = np.exp(g.random((topk, T), dtype=np.float32))
    return ids, (raw / raw.sum(axis=0, keepdims=True)).astype(np.float16)


@pytest.mark.parametrize("T,H,E,topk", [(256, 1024, 32, 2), (48, 512, 64, 8), (4096, 1024, 32, 2), (7, 64, 40, 3)])
def test_router_bit_exact(cuda, T, H, E, topk):
    import torch
    d = inputs.moe(tokens=T, hidden=H, experts=E, inter=8, topk=topk, seed=4)
    w, ids, logits = cuda.moe.moe_router(torch.from_numpy(d["X"]).cuda(), torch.from_numpy(d["Wr"]).cuda(), topk,
                                         return_logits=True)
    rids, rgates, rlogits = ref.moe_router(d["X"], d["Wr"], topk)
    assert np.array_equal(logits.cpu().numpy().view(np.uint32), rlogits.view(np.uint32))  # same f32 bits
    assert np.array_equal(ids.cpu().numpy(), rids)
    ulp = np.abs(w.cpu().numpy().view(np.int16).astype(np.int32) - rgates.view(np.int16).astype(np.int32))
    assert ulp.max() <= 1


# one token, hidden sizes off the 256-element chunks, several groups of tokens per CTA, experts that are no multiple of what a
# warp carries, router weights that do not fit in shared memory
@pytest.mark.parametrize("T,H,E,topk", [(1, 8, 3, 3), (300, 264, 35, 5), (700, 72, 33, 1), (5000, 264, 36, 4), (1300, 1544, 100, 2)])
def test_router_group_shapes(cuda, T, H, E, topk):
    test_router_bit_exact(cuda, T, H, E, topk)


def test_router_tie_goes_to_smallest_index(cuda):
    import torch
    X = np.zeros((3, 64), np.float16); X[:, 0] = 1
    Wr = np.zeros((16, 64), np.float16); Wr[[3, 5, 9], 0] = 2.0  # three equal maxima, the rest tie at 0
    w, ids = cuda.moe.moe_router(torch.from_numpy(X).cuda(), torch.from_numpy(Wr).cuda(), 4)
    assert ids.cpu().numpy()[:, 0].tolist() == [4, 6, 10, 1]


@pytest.mark.parametrize("T,E,topk,tile_m,dtype", [(48, 64, 8, 128, np.int64), (128, 32, 4, 128, np.int64),
                                                   (64, 64, 8, 128, np.int32), (256, 32, 2, 128, np.int32),
                                                   (4096, 32, 2, 128, np.int32), (1000, 7, 3, 16, np.int64),
                                                   (1, 4, 1, 32, np.int32)])
def test_align_bit_exact(cuda, T, E, topk, tile_m, dtype):
    import torch
    ids, _ = random_routing(T, E, topk, seed=T + E)
    tok, exp = cuda.moe.moe_align_tile_size(torch.from_numpy(ids.astype(dtype)).cuda(), tile_m, E)
    rtok, rexp = ref.moe_align_tile_size(ids, tile_m, E)
    assert np.array_equal(tok.cpu().numpy(), rtok)
    assert np.array_equal(exp.cpu().numpy(), rexp)


def test_align_skewed_and_empty_experts(cuda):
    import torch
    ids = np.ones((2, 300), np.int32); ids[1] = 5  # every token picks experts 1 and 5 only
    tok, exp = cuda.moe.moe_align_tile_size(torch.from_numpy(ids).cuda(), 128, 8)
    rtok, rexp = ref.moe_align_tile_size(ids, 128, 8)
    assert np.array_equal(tok.cpu().numpy(), rtok) and np.array_equal(exp.cpu().numpy(), rexp)
    bad = ids.copy(); bad[0, 7] = 9  # expert id out of range is reported, not silently used
    with pytest.raises(cuda.CtbError):
        cuda.moe.moe_align_tile_size(torch.from_numpy(bad).cuda(), 128, 8)


def dev(d, *names):
    import torch
    return [torch.from_numpy(d[n]).cuda() for n in names]


# examples/moe.jl:402-410 main() cases (random routing as in its prepare())
# the reference's main() cases, then cases with some hundred slots per expert: several full blocks per expert, ragged
# last blocks, an intermediate size that is not a multiple of the tile
@pytest.mark.parametrize("T,H,E,I,topk", [(48, 512, 64, 1024, 8), (128, 512, 32, 1024, 4), (64, 1024, 64, 2048, 8),
                                          (1024, 256, 4, 384, 2), (600, 512, 2, 256, 1), (1500, 320, 5, 136, 1)])
def test_cutile_moe_reference_cases(cuda, T, H, E, I, topk):
    import torch
    d = inputs.moe(tokens=T, hidden=H, experts=E, inter=I, topk=topk, seed=4)
    ids, w = random_routing(T, E, topk, seed=1)
    X, w1, w2 = dev(d, "X", "w1", "w2")
    out = cuda.moe.cutile_moe(X, w1, w2, torch.from_numpy(w).cuda(), torch.from_numpy(ids).cuda(), 128, 128, 64)
    torch.cuda.synchronize()
    want = ref.moe_ffn(d["X"], d["w1"], d["w2"], w, ids)
    assert ref.rel_fro(out.cpu().numpy(), want) <= TOL


# More than 2048 slots.  Blocks of one and of two MMAs whose accumulators follow each other in the ring of TMEM columns: experts at
# the edges of 256, 320 and 512 slots, and in turn with small ones; then token rows that do and do not fit a CTA of the sort at
# once, that fit only through registers, and more slots than a CTA counts itself.
@pytest.mark.parametrize("H,I,topk,counts", [
    (128, 2048, 1, (257, 320, 16, 272, 304, 0, 288, 321, 1, 319, 256, 255, 273, 17, 512, 513, 640, 289, 32, 320, 320, 320, 258)),
    (64, 1536, 1, (320, 33, 320, 320, 304, 304, 304, 16, 300, 1, 320, 320, 48, 290, 290, 290, 290, 700, 452, 226)),
    (8, 256, 3, 900), (16392, 16, 1, 2100), (41000, 8, 8, 257), (64, 64, 2, 8300)])
def test_cutile_moe_many_slots(cuda, H, I, topk, counts):
    import torch
    g = np.random.default_rng(11)
    if topk == 1 and isinstance(counts, tuple):
        ids = g.permutation(np.repeat(np.arange(len(counts)), counts))[None] + 1
        T, E = ids.shape[1], len(counts)
        w = g.random((1, T)).astype(np.float16)
    else:
        T, E = counts, 9 if topk < 8 else 8
        ids, w = random_routing(T, E, topk, seed=3)
    d = inputs.moe(tokens=T, hidden=H, experts=E, inter=I, topk=topk, seed=6)
    X, w1, w2 = dev(d, "X", "w1", "w2")
    out = cuda.moe.cutile_moe(X, w1, w2, torch.from_numpy(w).cuda(), torch.from_numpy(ids.astype(np.int32)).cuda(), 128, 128, 64)
    again = cuda.moe.cutile_moe(X, w1, w2, torch.from_numpy(w).cuda(), torch.from_numpy(ids.astype(np.int64)).cuda(), 128, 128, 64)
    assert torch.equal(out, again)
    want = ref.moe_ffn(d["X"], d["w1"], d["w2"], w, ids)
    assert ref.rel_fro(out.cpu().numpy(), want) <= TOL


FIRST_CALL = """
import sys
import numpy as np
import torch
import cutile_b200 as ctb
from oracle import inputs, ref
from test_moe_gpu import TOL, dev, random_routing
T, H, E, topk = map(int, sys.argv[1:])
d = inputs.moe(tokens=T, hidden=H, experts=E, inter=16, topk=topk, seed=4)
ids, w = random_routing(T, E, topk, seed=1)
X, w1, w2 = dev(d, "X", "w1", "w2")
want = ref.moe_ffn(d["X"], d["w1"], d["w2"], w, ids)
for dtype in (np.int32, np.int64):
    out = ctb.moe.cutile_moe(X, w1, w2, torch.from_numpy(w).cuda(), torch.from_numpy(ids.astype(dtype)).cuda(), 128, 128, 64)
    assert ref.rel_fro(out.cpu().numpy(), want) <= TOL
"""


# The sort's shared memory is between 48 KB less its static part and 48 KB (22 token rows of 2 KB and the counts of 32 experts; 8 of
# 5760 bytes), and no larger call of the process has raised the limit before: a process of its own.
@pytest.mark.parametrize("T,H,E,topk", [(3000, 1024, 32, 2), (950, 2880, 32, 4)])
def test_cutile_moe_first_call_of_a_process(cuda, T, H, E, topk):
    import os
    import subprocess
    import sys
    here = os.path.dirname(os.path.abspath(__file__))
    root = os.path.dirname(here)
    env = dict(os.environ, PYTHONPATH=os.pathsep.join([root, os.path.join(root, "cutile.jl_b200"), here]))
    r = subprocess.run([sys.executable, "-c", FIRST_CALL, *map(str, (T, H, E, topk))], capture_output=True, text=True, timeout=300, env=env)
    assert r.returncode == 0, r.stderr[-2000:]


def test_moe_benchmark_config_with_router(cuda):
    import torch
    d = inputs.moe()  # 256 tokens, hidden 1024, 32 experts, inter 2048, top-2, seed 4
    X, Wr, w1, w2 = dev(d, "X", "Wr", "w1", "w2")
    w, ids = cuda.moe.moe_router(X, Wr, 2)
    out = cuda.moe.cutile_moe(X, w1, w2, w, ids, 128, 128, 64)
    torch.cuda.synchronize()
    rids, rgates, _ = ref.moe_router(d["X"], d["Wr"], 2)
    assert np.array_equal(ids.cpu().numpy(), rids)
    want = ref.moe_ffn(d["X"], d["w1"], d["w2"], rgates, rids)
    assert ref.rel_fro(out.cpu().numpy(), want) <= TOL
    out2 = cuda.moe.cutile_moe(X, w1, w2, w, ids, 128, 128, 64)
    assert torch.equal(out, out2)  # no atomics anywhere: bitwise repeatable


def test_moe_three_kernel_path_matches_reference_structure(cuda):
    """The reference's own decomposition (examples/moe.jl:228-256): grouped GEMM -> SiLU*mul -> grouped GEMM with
    routing weights -> sum over slots, through the per-kernel entry points."""
    import torch
    T, H, E, I, topk = 96, 256, 16, 512, 4
    d = inputs.moe(tokens=T, hidden=H, experts=E, inter=I, topk=topk, seed=8)
    ids, w = random_routing(T, E, topk, seed=2)
    X, w1, w2 = dev(d, "X", "w1", "w2")
    tok, exp = cuda.moe.moe_align_tile_size(torch.from_numpy(ids).cuda(), 64, E)
    total = T * topk
    cache1 = torch.zeros(total, 2 * I, device="cuda", dtype=torch.float16)
    cache2 = torch.zeros(total, I, device="cuda", dtype=torch.float16)
    cache3 = torch.zeros(total, H, device="cuda", dtype=torch.float16)
    wflat = torch.from_numpy(np.ascontiguousarray(w.T).reshape(-1)).cuda()  # vec(permutedims(topk_weights))
    cuda.moe.fused_moe_kernel(X, w1, cache1, wflat, tok, exp, topk, False, 64, 128, 64)
    cuda.moe.silu_and_mul_kernel(cache1[:, :I], cache1[:, I:], cache2, 512)
    cuda.moe.fused_moe_kernel(cache2, w2, cache3, wflat, tok, exp, 1, True, 64, 128, 64)
    out = cache3.view(T, topk, H).float().sum(dim=1)
    torch.cuda.synchronize()
    want = ref.moe_ffn(d["X"], d["w1"], d["w2"], w, ids)
    assert ref.rel_fro(out.cpu().numpy(), want) <= 3e-3  # three f16 roundings of intermediates, as in the reference
    fused = cuda.moe.cutile_moe(X, w1, w2, torch.from_numpy(w).cuda(), torch.from_numpy(ids).cuda(), 64, 128, 64)
    assert ref.rel_fro(fused.cpu().numpy(), want) <= TOL


def test_moe_full_size_token_permutation(cuda):
    """4096-token configuration: a token's output depends only on its own row and routing, so permuting the tokens
    permutes the output bit for bit; a 256-token sample is also checked against the oracle."""
    import torch
    d = inputs.moe(tokens=4096, seed=4)
    X, Wr, w1, w2 = dev(d, "X", "Wr", "w1", "w2")
    w, ids = cuda.moe.moe_router(X, Wr, 2)
    out = cuda.moe.cutile_moe(X, w1, w2, w, ids, 128, 128, 64)
    perm = torch.randperm(4096, device="cuda", generator=torch.Generator(device="cuda").manual_seed(0))
    outp = cuda.moe.cutile_moe(X[perm].contiguous(), w1, w2, w[:, perm].contiguous(), ids[:, perm].contiguous(),
                               128, 128, 64)
    assert torch.equal(outp, out[perm])
    sample = np.arange(0, 4096, 16)
    idn, wn = ids.cpu().numpy(), w.cpu().numpy()
    want = ref.moe_ffn(d["X"][sample], d["w1"], d["w2"], wn[:, sample], idn[:, sample])
    assert ref.rel_fro(out.cpu().numpy()[sample], want) <= TOL


def test_moe_rejections(cuda):
    import torch
    lib = cuda._lib
    d = inputs.moe(tokens=8, hidden=64, experts=4, inter=64, topk=2, seed=1)
    X, w1, w2 = dev(d, "X", "w1", "w2")
    ids, w = random_routing(8, 4, 2, 0)
    idd, wd = torch.from_numpy(ids).cuda(), torch.from_numpy(w).cuda()
    with pytest.raises(cuda.CtbError) as e:
        cuda.moe.cutile_moe(X, w1, w2, wd, idd, 100, 128, 64)
    assert e.value.status == lib.UNSUPPORTED_TILE
    with pytest.raises(cuda.CtbError) as e:
        cuda.moe.cutile_moe(X, w1, w2[:, :, :32].contiguous(), wd, idd, 128, 128, 64)
    assert e.value.status == lib.BAD_ARG


# slots per expert around the block sizes: one slot, 16, 17, up to 256 (one block), 257 and more (two, three blocks), one
# expert with everything, empty experts, row counts off the 128- and 256-row tiles, a reduction length off the k-block,
# more slots than a CTA of the sort counts itself
@pytest.mark.parametrize("T,H,E,I,topk,skew", [(1, 64, 4, 64, 1, False), (1, 512, 64, 1024, 8, False), (17, 128, 3, 200, 1, True),
                                               (257, 264, 2, 72, 1, True), (300, 512, 5, 136, 2, False), (700, 72, 1, 320, 1, False),
                                               (640, 512, 16, 256, 4, True), (3, 1024, 256, 128, 8, False), (5000, 64, 7, 64, 4, False)])
@pytest.mark.parametrize("ids64", [False, True])
def test_cutile_moe_block_shapes(cuda, T, H, E, I, topk, skew, ids64):
    import torch
    d = inputs.moe(tokens=T, hidden=H, experts=E, inter=I, topk=topk, seed=6)
    ids, w = random_routing(T, E, topk, seed=T)
    if skew:  # most tokens choose the first expert (first choices only: a token's choices stay different)
        first = np.where(np.arange(T) % 8 < 7, 1, ids[0])
        clash = (ids == 1) & (np.arange(topk)[:, None] > 0) & (first == 1)
        ids = np.where(clash, ids[0][None, :], ids)
        ids[0] = first
    X, w1, w2 = dev(d, "X", "w1", "w2")
    args = (X, w1, w2, torch.from_numpy(w).cuda(), torch.from_numpy(ids if ids64 else ids.astype(np.int32)).cuda(), 128, 128, 64)
    out, again = cuda.moe.cutile_moe(*args), cuda.moe.cutile_moe(*args)
    assert torch.equal(out, again)
    want = ref.moe_ffn(d["X"], d["w1"], d["w2"], w, ids)
    assert ref.rel_fro(out.cpu().numpy(), want) <= TOL
    cuda.check_device_status(0)


def test_cutile_moe_bad_expert_id_is_reported(cuda):
    import torch
    d = inputs.moe(tokens=40, hidden=64, experts=4, inter=64, topk=2, seed=1)
    ids, w = random_routing(40, 4, 2, 0)
    ids[1, 7] = 5
    X, w1, w2 = dev(d, "X", "w1", "w2")
    cuda.moe.cutile_moe(X, w1, w2, torch.from_numpy(w).cuda(), torch.from_numpy(ids).cuda(), 128, 128, 64)
    with pytest.raises(cuda.CtbError):
        cuda.check_device_status(0)
    ids[1, 7] = 1 + ids[0, 7] % 4
    out = cuda.moe.cutile_moe(X, w1, w2, torch.from_numpy(w).cuda(), torch.from_numpy(ids).cuda(), 128, 128, 64)
    assert ref.rel_fro(out.cpu().numpy(), ref.moe_ffn(d["X"], d["w1"], d["w2"], w, ids)) <= TOL

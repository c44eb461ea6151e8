"""GPU parity of the flash-attention forward kernel against the float64 oracle.

Tolerance: relative Frobenius error <= 2e-3 (f16 operands, f32 softmax state and
accumulation, f16 output).  The reference's own check is norm-wise rtol=1e-2,
atol=1e-3 (examples/fmha.jl:277-282)."""
import numpy as np
import pytest

from oracle import inputs, ref

pytestmark = pytest.mark.gpu
TOL = 2e-3


def run(cuda, d, **kw):
    import torch
    Q, K, V = (torch.from_numpy(d[k]).cuda() for k in ("Q", "K", "V"))
    out = cuda.fmha.cutile_fmha(Q, K, V, **kw)
    torch.cuda.synchronize()
    return out.cpu().numpy()


# examples/fmha.jl:314-325 main() cases, then the benchmark shape
@pytest.mark.parametrize("batch,heads,seq,causal", [(2, 8, 128, False), (2, 8, 128, True), (4, 16, 256, True),
                                                    (8, 16, 1024, True), (1, 2, 1024, False)])
def test_fmha_reference_cases(cuda, batch, heads, seq, causal):
    d = inputs.fmha(batch, heads, seq, seq, 64, seed=3)
    out = run(cuda, d, causal=causal)
    want = ref.fmha(d["Q"], d["K"], d["V"], causal=causal)
    assert out.dtype == np.float16
    assert ref.rel_fro(out, want) <= TOL
    err = np.linalg.norm(out.astype(np.float64) - want)
    assert err <= max(1e-3, 1e-2 * np.linalg.norm(want))  # the reference's own criterion


@pytest.mark.parametrize("seq_q,seq_kv,causal,input_pos,heads,kv_heads", [
    (200, 300, False, 0, 4, 4),    # ragged Q and K tiles (EVEN_K false)
    (200, 200, True, 0, 4, 4),     # ragged + causal
    (128, 384, True, 256, 4, 4),   # prefill with a cache: queries sit at positions 256..383
    (100, 333, True, 233, 2, 2),   # ragged everything with an offset
    (256, 256, True, 0, 8, 2),     # grouped-query attention, group of 4
    (256, 512, False, 0, 6, 3),    # GQA, non-causal, rectangular
    (1, 1, True, 0, 1, 1),         # a single query and key
])
def test_fmha_options(cuda, seq_q, seq_kv, causal, input_pos, heads, kv_heads):
    d = inputs.fmha(2, heads, seq_q, seq_kv, 64, kv_heads=kv_heads, seed=13)
    out = run(cuda, d, causal=causal, input_pos=input_pos, query_group_size=heads // kv_heads)
    want = ref.fmha(d["Q"], d["K"], d["V"], causal=causal, input_pos=input_pos)
    assert ref.rel_fro(out, want) <= TOL
    for h in range(heads):  # per head, so that a wrong KV-head mapping cannot hide in the norm
        assert ref.rel_fro(out[:, h], want[:, h]) <= TOL


def test_fmha_scale_and_large_scores(cuda):
    d = inputs.fmha(1, 2, 256, 256, 64, seed=21)
    d["Q"] = (d["Q"].astype(np.float32) * 6).astype(np.float16)  # sharp softmax: exercises the running max
    out = run(cuda, d, causal=True, qk_scale=0.3)
    want = ref.fmha(d["Q"], d["K"], d["V"], qk_scale=0.3, causal=True)
    assert ref.rel_fro(out, want) <= TOL


# (batch, kv heads, group, query rows, keys): one pair in as many parts as SMs, parts of unequal length, two parts, one part each, as
# many pairs as SMs and one more, pairs that leave half of the SMs idle in parts (long: ranges), more pairs than SMs in ranges of
# blocks and of whole pairs (twice as many, and a few more), 1 to 16 rows
@pytest.mark.parametrize("batch,kvh,group,seq_q,keys", [
    (1, 1, 1, 1, 40000), (1, 1, 4, 4, 300), (1, 3, 1, 9, 5000), (2, 37, 2, 4, 513), (5, 10, 8, 1, 900), (3, 19, 3, 3, 9 * 256),
    (75, 1, 1, 1, 1024), (75, 1, 1, 1, 9000), (37, 4, 1, 1, 600), (149, 1, 3, 1, 600), (1, 2, 16, 1, 257),
    (160, 1, 1, 1, 3000), (150, 2, 1, 3, 900), (74, 4, 2, 2, 700), (74, 4, 16, 1, 1100)])
@pytest.mark.parametrize("dtype", ["float16", "bfloat16"])
def test_fmha_few_rows_parts(cuda, dtype, batch, kvh, group, seq_q, keys):
    import torch
    g = torch.Generator(device="cuda").manual_seed(keys)
    dt = getattr(torch, dtype)
    q, k, v = (torch.randn(batch, h, n, 64, device="cuda", generator=g).to(dt)
               for h, n in ((kvh * group, seq_q), (kvh, keys), (kvh, keys)))
    out = cuda.fmha.cutile_fmha(q, k, v, causal=True, input_pos=keys - seq_q, query_group_size=group)
    assert torch.equal(out, cuda.fmha.cutile_fmha(q, k, v, causal=True, input_pos=keys - seq_q, query_group_size=group))
    for b in range(batch):
        s = q[b].double() @ k[b].double().repeat_interleave(group, 0).transpose(1, 2) / 8
        s.masked_fill_(torch.arange(keys, device="cuda") > torch.arange(seq_q, device="cuda")[:, None] + keys - seq_q, -torch.inf)
        want = torch.softmax(s, -1) @ v[b].double().repeat_interleave(group, 0)
        assert (out[b] - want).norm() <= (TOL if dtype == "float16" else 1e-2) * want.norm()


def grouped(q, k, v, cuts):
    """Attention of one query position over pairs [P, heads or 1, keys, 64], in f64 but for the probabilities, which are rounded to
    the type of v relative to a running maximum: of every 32 keys of each 256, from one of `cuts` (blocks of 256 keys, counted
    over all pairs) to the next."""
    import torch
    P, H, keys = q.shape[0], q.shape[1], k.shape[2]
    n = -(-keys // 256)
    s = torch.full((P, H, n * 256), -torch.inf, device="cuda", dtype=torch.float64)
    s[..., :keys] = (q.double() @ k.double().transpose(2, 3))[:, :, 0] * (0.125 * 1.4426950408889634)
    s = s.view(P, H, n, 8, 32).permute(2, 0, 3, 1, 4)
    w = torch.zeros(P, n * 256, 64, device="cuda", dtype=torch.float64)
    w[:, :keys] = v[:, 0].double()
    w = w.view(P, n, 8, 32, 64).permute(1, 0, 2, 3, 4)
    first = torch.zeros(P * n, dtype=torch.bool, device="cuda")
    first[torch.tensor(sorted(c for c in cuts if c < P * n), device="cuda")] = True
    first = first.view(P, n)
    shape = (P, 8, H, 1)
    M, L, O = torch.full(shape, -torch.inf, device="cuda").double(), torch.zeros(shape, device="cuda").double(), 0.0
    m, l, o = M.clone(), L.clone(), torch.zeros(P, 8, H, 64, device="cuda").double()

    def merge(M, L, O, m, l, o):
        top = torch.maximum(M, m)
        f, g = (torch.exp2(x - torch.where(top == -torch.inf, 0.0, top)) for x in (M, m))
        return top, L * f + l * g, O * f + o * g
    for j in range(n):
        new = first[:, j].view(P, 1, 1, 1)
        M2, L2, O2 = merge(M, L, O, m, l, o)
        M, L, O = torch.where(new, M2, M), torch.where(new, L2, L), torch.where(new, O2, O + torch.zeros_like(o))
        m, l, o = torch.where(new, -torch.inf, m), torch.where(new, 0.0, l), torch.where(new, 0.0, o)
        top = torch.maximum(m, s[j].amax(-1, keepdim=True))
        ref = torch.where(top == -torch.inf, 0.0, top)
        p, f = torch.exp2(s[j] - ref), torch.exp2(m - ref)
        m, l, o = top, l * f + p.sum(-1, keepdim=True), o * f + p.to(v.dtype).double() @ w[j]
    M, L, O = merge(M, L, O, m, l, o)
    f = torch.exp2(M - M.amax(1, keepdim=True))
    return ((O * f).sum(1) / (L * f).sum(1)).view(P, H, 1, 64).to(v.dtype)


# What is rounded to 16 bits is rounded as in equal ranges of blocks, one per SM, whatever a CTA works through: whole pairs (twice),
# one part of a pair (cut once, twice), two parts, ranges.  Another grouping changes 14 to 31 % of the outputs.  With the same one the
# kernel's probabilities are off by about 1e-6 (f32 scores times log2(e), approximate exponential), so of 4000 in f16 (half a step:
# 2.4e-4 to 4.9e-4) a dozen are rounded the other way; each moves an output by 2^-11 / 4000 = 1.2e-7, all of them by 4e-7, and a step of
# an output of 0.02 is 1e-5: 4 % of the outputs come out otherwise.  In bf16 it is one of 4000, 1e-6 against 8e-5: 1 %.
@pytest.mark.parametrize("pairs,heads,keys", [(256, 4, 4000), (200, 16, 900), (100, 1, 2000), (75, 4, 1000), (64, 4, 2000), (160, 1, 3000)])
@pytest.mark.parametrize("dtype", ["float16", "bfloat16"])
def test_fmha_few_rows_grouping(cuda, dtype, pairs, heads, keys):
    import torch
    g = torch.Generator(device="cuda").manual_seed(keys)
    q, k, v = (torch.randn(pairs, h, n, 64, device="cuda", generator=g).to(getattr(torch, dtype))
               for h, n in ((heads, 1), (1, keys), (1, keys)))
    sms, n = torch.cuda.get_device_properties(0).multi_processor_count, -(-keys // 256)
    cuts = {c * pairs * n // sms for c in range(sms)} | set(range(0, pairs * n, n))
    for k0 in range(1, min(n, sms // pairs) if pairs <= sms else 1):  # equal parts
        cuts |= {pr * n + k0 * n // min(n, sms // pairs) for pr in range(pairs)}
    out = cuda.fmha.cutile_fmha(q, k, v, causal=True, input_pos=keys - 1, query_group_size=heads)
    assert (out != grouped(q, k, v, cuts)).double().mean() < (0.08 if dtype == "float16" else 0.02)


def test_fmha_causal_prefix_property_full_size(cuda):
    """Size-independent property at the benchmark shape: under the causal mask the output of the first 512
    queries does not depend on the later keys/values, so it equals the result on the truncated problem."""
    import torch
    g = torch.Generator(device="cuda").manual_seed(3)
    Q, K, V = (torch.randn(8, 16, 1024, 64, device="cuda", generator=g).half() for _ in range(3))
    full = cuda.fmha.cutile_fmha(Q, K, V, causal=True)
    half = cuda.fmha.cutile_fmha(Q[:, :, :512].contiguous(), K[:, :, :512].contiguous(), V[:, :, :512].contiguous(),
                                 causal=True)
    assert torch.equal(full[:, :, :512], half)
    assert torch.isfinite(full).all()


def test_fmha_rejections(cuda):
    import torch
    lib = cuda._lib
    q = torch.zeros(1, 2, 128, 64, device="cuda", dtype=torch.float16)
    with pytest.raises(cuda.CtbError) as e:
        cuda.fmha.cutile_fmha(q, q, q, tile_m=96)
    assert e.value.status == lib.UNSUPPORTED_TILE
    with pytest.raises(cuda.CtbError) as e:
        cuda.fmha.cutile_fmha(q, q, q, query_group_size=3)
    assert e.value.status == lib.BAD_ARG
    q32 = torch.zeros(1, 2, 128, 32, device="cuda", dtype=torch.float16)
    with pytest.raises(cuda.CtbError) as e:
        cuda.fmha.cutile_fmha(q32, q32, q32)
    assert e.value.status == lib.UNSUPPORTED


@pytest.mark.parametrize("batch,heads,seq_q,seq_kv,causal,input_pos,kv_heads", [
    (2, 8, 128, 128, True, 0, 8), (8, 16, 1024, 1024, True, 0, 16), (2, 4, 200, 333, True, 133, 2), (1, 2, 256, 512, False, 0, 2)])
def test_fmha_bf16(cuda, batch, heads, seq_q, seq_kv, causal, input_pos, kv_heads):
    """bfloat16 operands (examples/fmha.jl takes the element type as a parameter, :236): the same kernel with bf16 MMAs,
    probabilities and output rounded to bf16.  The oracle is fed the bf16-rounded inputs; tolerance 1e-2 (8 mantissa
    bits in P and in the output)."""
    import torch
    d = inputs.fmha(batch, heads, seq_q, seq_kv, 64, kv_heads=kv_heads, seed=17)
    Q, K, V = (torch.from_numpy(d[k].astype(np.float32)).cuda().to(torch.bfloat16) for k in ("Q", "K", "V"))
    out = cuda.fmha.cutile_fmha(Q, K, V, causal=causal, input_pos=input_pos, query_group_size=heads // kv_heads)
    torch.cuda.synchronize()
    assert out.dtype == torch.bfloat16
    back = lambda t: t.float().cpu().numpy()
    want = ref.fmha(back(Q), back(K), back(V), causal=causal, input_pos=input_pos)
    assert ref.rel_fro(back(out), want) <= 1e-2
    cuda.check_device_status(0)


@pytest.mark.parametrize("batch,heads,kv_heads,seq_q,seq_kv,causal,input_pos", [
    (1, 1, 1, 1, 1, True, 0), (2, 8, 2, 1, 31, True, 30), (3, 16, 2, 1, 256, True, 255), (1, 32, 4, 1, 257, True, 256),
    (5, 4, 4, 1, 1000, True, 999), (1, 8, 8, 1, 8191, True, 8190), (2, 16, 1, 1, 3000, True, 2999), (2, 16, 4, 4, 700, True, 696),
    (1, 5, 5, 16, 333, True, 317), (2, 6, 3, 8, 64, True, 0), (2, 8, 4, 3, 500, False, 0), (1, 4, 4, 1, 900, True, 200),
    (40, 8, 4, 1, 2049, True, 2048)])
@pytest.mark.parametrize("bf16", [False, True])
def test_fmha_decode(cuda, batch, heads, kv_heads, seq_q, seq_kv, causal, input_pos, bf16):
    """Few query rows per key/value head: 1, up to 8 and up to 16 rows, keys in one block, at block edges, over several
    CTAs and with several pairs per CTA, keys behind the last visible one, twice in a row (the arrival counters are back at
    zero, the order of summation is fixed)."""
    import torch
    dt = torch.bfloat16 if bf16 else torch.float16
    d = inputs.fmha(batch, heads, seq_q, seq_kv, 64, kv_heads=kv_heads, seed=19)
    Q, K, V = (torch.from_numpy(d[k].astype(np.float32)).cuda().to(dt) for k in ("Q", "K", "V"))
    run = lambda: cuda.fmha.cutile_fmha(Q, K, V, causal=causal, input_pos=input_pos, query_group_size=heads // kv_heads)
    out, again = run(), run()
    assert torch.equal(out, again)
    back = lambda t: t.float().cpu().numpy()
    want = ref.fmha(back(Q), back(K), back(V), causal=causal, input_pos=input_pos)
    for h in range(heads):
        assert ref.rel_fro(back(out)[:, h], want[:, h]) <= (1e-2 if bf16 else TOL)
    cuda.check_device_status(0)


@pytest.mark.parametrize("heads,kv_heads,seq_q,seq_kv,input_pos", [
    (8, 2, 1, 900, 200), (8, 8, 1, 256, 127), (4, 4, 1, 64, 0), (16, 4, 4, 1000, 380), (5, 5, 16, 700, 256),
    (4, 4, 100, 500, 30), (8, 2, 200, 1000, 333), (1184, 1184, 10, 200, 90)])  # two with 128-row tiles, many heads
@pytest.mark.parametrize("bf16", [False, True])
def test_fmha_unwritten_cache(cuda, heads, kv_heads, seq_q, seq_kv, input_pos, bf16):
    """Rows of a preallocated cache behind the last visible key are never written by the caller: whatever lies there (NaN and
    infinities included) stays out of the result, which equals that of a cache that ends at the last visible key."""
    import torch
    dt = torch.bfloat16 if bf16 else torch.float16
    d = inputs.fmha(2, heads, seq_q, seq_kv, 64, kv_heads=kv_heads, seed=23)
    Q, K, V = (torch.from_numpy(d[k].astype(np.float32)).cuda().to(dt) for k in ("Q", "K", "V"))
    n = input_pos + seq_q
    run = lambda k, v: cuda.fmha.cutile_fmha(Q, k, v, causal=True, input_pos=input_pos, query_group_size=heads // kv_heads)
    want = run(K[:, :, :n].contiguous(), V[:, :, :n].contiguous())
    for bad in (float("nan"), float("inf"), float("-inf")):
        K[:, :, n:], V[:, :, n:] = bad, bad
        assert torch.equal(run(K, V), want)
    cuda.check_device_status(0)


@pytest.mark.parametrize("batch,heads,seq_q,seq_kv", [(3, 800, 16, 100), (2, 1184, 9, 33), (2, 1184, 16, 256), (2, 1184, 16, 257),
                                                     (2, 1184, 16, 32), (4, 600, 8, 100), (100, 16, 12, 12)])
def test_fmha_many_short_heads(cuda, batch, heads, seq_q, seq_kv):
    """Few rows, few keys, many heads: warps without keys, several heads per CTA and Q of the next."""
    d = inputs.fmha(batch, heads, seq_q, seq_kv, 64, seed=29)
    out = run(cuda, d, causal=True, input_pos=seq_kv - seq_q)
    want = ref.fmha(d["Q"], d["K"], d["V"], causal=True, input_pos=seq_kv - seq_q)
    assert ref.rel_fro(out, want) <= TOL
    cuda.check_device_status(0)

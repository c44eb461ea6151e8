"""GPU parity of the LayerNorm kernels against the float64 oracle.

Tolerance (f32): max|out-ref| / max|ref| <= 1e-5 for Y, dX, Mean, Rstd, dW, dB
(the reference's own check is norm-wise rtol=1e-2, examples/layernorm.jl:300-312)."""
import numpy as np
import pytest

from oracle import inputs, ref

pytestmark = pytest.mark.gpu
TOL = 1e-5


def run_fwd_bwd(cuda, d, G=64, ld=None):
    import torch
    ln = cuda.layernorm
    M, N = d["M"], d["N"]
    ld = ld or N
    def dev2d(a):
        t = torch.zeros(M, ld, device="cuda")
        t[:, :N] = torch.from_numpy(a).cuda()
        return t[:, :N]
    X, DY = dev2d(d["X"]), dev2d(d["DY"])
    W, B = torch.from_numpy(d["W"]).cuda(), torch.from_numpy(d["B"]).cuda()
    Y = torch.zeros(M, ld, device="cuda")[:, :N]
    DX = torch.zeros(M, ld, device="cuda")[:, :N]
    Mean, Rstd = torch.empty(M, device="cuda"), torch.empty(M, device="cuda")
    DWp = torch.full((G, N), float("nan"), device="cuda")  # never zero-filled: must be fully overwritten
    DBp = torch.full((G, N), float("nan"), device="cuda")
    FDW, FDB = torch.empty(N, device="cuda"), torch.empty(N, device="cuda")
    ln.layer_norm_fwd(X, W, B, Y, Mean, Rstd, float(d["eps"]), 1024)
    ln.layer_norm_bwd_dx_partial_dwdb(DX, DY, DWp, DBp, X, W, Mean, Rstd, None, G, 1024)
    ln.layer_norm_bwd_dwdb(DWp, DBp, FDW, FDB, 32, 1024)
    torch.cuda.synchronize()
    return [t.cpu().numpy() for t in (Y, Mean, Rstd, DX, FDW, FDB)]


# the reference's main() cases (examples/layernorm.jl:340-348), the benchmark
# shape, ragged/odd shapes (generic path), wide rows, fewer rows than groups.
@pytest.mark.parametrize("M,N,G", [(256, 256, 64), (512, 512, 64), (1024, 1024, 64), (4096, 4096, 64),
                                   (37, 1000, 64), (5, 333, 8), (130, 8192, 16), (3, 2048, 64), (300, 4096, 1)])
def test_layernorm_parity(cuda, M, N, G):
    d = inputs.layernorm(M=M, N=N, seed=0)
    Y, Mean, Rstd, DX, DW, DB = run_fwd_bwd(cuda, d, G)
    rY, rMean, rRstd = ref.layernorm_fwd(d["X"], d["W"], d["B"], d["eps"])
    rDX, rDW, rDB = ref.layernorm_bwd(d["X"], d["W"], d["DY"], rMean, rRstd)
    for name, got, want in (("Y", Y, rY), ("Mean", Mean, rMean), ("Rstd", Rstd, rRstd), ("dX", DX, rDX),
                            ("dW", DW, rDW), ("dB", DB, rDB)):
        err = ref.max_abs_over_max(got, want)
        assert err <= TOL, (name, err)
        # element-wise relative error with the floor 1e-3 * max|ref| (pure relative error is unbounded where Y or dX
        # cross zero); measured 1e-6..1e-5 on these shapes
        assert ref.max_rel(got, want) <= 1e-3, (name, ref.max_rel(got, want))
        assert ref.rel_fro(got, want) <= 1e-2  # the reference's own criterion


# around the widths that change the kernel (256, 512, 1024, 2048, 4096, 8192 columns), on and off the 16-byte grid, with rows
# on both sides of the lines M = N and M = N / 4, fewer rows than groups or warps, a group count that is no power of two
@pytest.mark.parametrize("M,N,G", [(9, 5, 64), (700, 31, 64), (3, 255, 3), (1000, 260, 7), (130, 511, 64), (600, 512, 64),
                                   (127, 513, 2), (60, 516, 64), (1030, 1023, 64), (300, 1024, 64), (70, 1025, 64),
                                   (513, 2047, 16), (40, 2051, 64), (100, 4099, 64), (20, 8191, 5)])
def test_layernorm_row_widths(cuda, M, N, G):
    test_layernorm_parity(cuda, M, N, G)


# the backward kernel whose warps have rings of rows: no row, one, fewer and more rows per warp than stages, the widths where the
# rows per lane and the warps change, rows on both sides of the lines 1024 and 4096 below 256 columns
@pytest.mark.parametrize("M,N,G", [(66, 260, 64), (1500, 512, 8), (3100, 516, 64), (5000, 1024, 3), (4000, 1020, 64),
                                   (1025, 8, 64), (4096, 252, 64), (4097, 256, 64), (1024, 256, 64), (2000, 300, 200), (2000, 256, 32), (2000, 256, 31),
                                   (2000, 256, 149)])
def test_layernorm_row_rings(cuda, M, N, G):
    test_layernorm_parity(cuda, M, N, G)


# and the kernel without rings where that is expected to be faster: one to eight CTAs per group, more groups than SMs and than
# clusters that run at once
@pytest.mark.parametrize("M,N,G", [(9000, 260, 12), (4000, 512, 17), (2000, 768, 37), (5000, 640, 18), (1200, 1024, 200), (1200, 512, 300)])
def test_layernorm_rings_or_not(cuda, M, N, G):
    test_layernorm_parity(cuda, M, N, G)


# dW and dB against 64 bits, of forty draws each: no less exact than a warp's rows one by one, then eight warps and up to eight CTAs one
# by one, then the groups (f32 in that order, with the CTAs that the kernel without rings has per group).  The noise of the mean is
# about 1 %; sixteen warps one by one are 3 to 15 % off.
@pytest.mark.parametrize("M,N,G,ctas", [(2000, 512, 64, 2), (4000, 400, 64, 4), (4000, 256, 64, 4), (2000, 260, 16, 8), (5000, 768, 18, 8)])
def test_layernorm_bwd_precision(cuda, M, N, G, ctas):
    import torch
    g = torch.Generator(device="cuda").manual_seed(M + N)
    ours, chain = np.zeros(2), np.zeros(2)

    def one_by_one(t, dim):
        s = t.select(dim, 0)
        for k in range(1, t.shape[dim]):
            s = s + t.select(dim, k)
        return s
    for _ in range(40):
        x, dy = (torch.randn(M, N, device="cuda", generator=g) for _ in range(2))
        w, mean, rstd = torch.ones(N, device="cuda"), torch.empty(M, device="cuda"), torch.empty(M, device="cuda")
        y, dx, part = torch.empty_like(x), torch.empty_like(x), torch.empty(2, G, N, device="cuda")
        out = torch.empty(2, N, device="cuda")
        cuda.layernorm.layer_norm_fwd(x, w, w, y, mean, rstd, 1e-5, 1024)
        cuda.layernorm.layer_norm_bwd_dx_partial_dwdb(dx, dy, part[0], part[1], x, w, mean, rstd, None, G, 1024)
        cuda.layernorm.layer_norm_bwd_dwdb(part[0], part[1], out[0], out[1], 32, 1024)
        terms = torch.stack((dy * ((x - mean[:, None]) * rstd[:, None]), dy))
        exact = torch.stack(((dy.double() * ((x.double() - mean.double()[:, None]) * rstd.double()[:, None])).sum(0), dy.double().sum(0)))
        rows = -(-M // (G * ctas * 8))  # of a warp; row g + G (8 cta + warp + 8 ctas j)
        t = torch.zeros(2, rows * ctas * 8 * G, N, device="cuda")
        t[:, :M] = terms
        other = torch.empty(2, N, device="cuda")
        t = one_by_one(one_by_one(one_by_one(t.view(2, rows, ctas, 8, G, N), 1), 2), 1).contiguous()
        cuda.layernorm.layer_norm_bwd_dwdb(t[0], t[1], other[0], other[1], 32, 1024)
        for e, v in ((ours, out), (chain, other)):
            e += ((v.double() - exact).norm(dim=1) / exact.norm(dim=1)).cpu().numpy()
    assert (ours <= 1.02 * chain).all(), (ours / 40, chain / 40)


@pytest.mark.parametrize("M", [64, 700])
def test_layernorm_strided(cuda, M):
    d = inputs.layernorm(M=M, N=512, seed=5)
    Y, Mean, Rstd, DX, DW, DB = run_fwd_bwd(cuda, d, 64, ld=640)
    rY, rMean, rRstd = ref.layernorm_fwd(d["X"], d["W"], d["B"], d["eps"])
    rDX, rDW, rDB = ref.layernorm_bwd(d["X"], d["W"], d["DY"], rMean, rRstd)
    assert ref.max_abs_over_max(Y, rY) <= TOL and ref.max_abs_over_max(DX, rDX) <= TOL
    assert ref.max_abs_over_max(DW, rDW) <= TOL and ref.max_abs_over_max(DB, rDB) <= TOL


def test_layernorm_bwd_is_deterministic(cuda):
    d = inputs.layernorm(M=2048, N=4096, seed=3)
    a = run_fwd_bwd(cuda, d)
    b = run_fwd_bwd(cuda, d)
    for x, y in zip(a, b):
        assert np.array_equal(x, y)  # lock-free fixed-order reduction: bitwise repeatable


def test_layernorm_rejections(cuda):
    import torch
    lib = cuda._lib
    X = torch.zeros(4, 256, device="cuda")
    v = torch.zeros(256, device="cuda"); m = torch.zeros(4, device="cuda")
    with pytest.raises(cuda.CtbError) as e:
        cuda.layernorm.layer_norm_fwd(X, v, v, torch.empty_like(X), m, m.clone(), 1e-5, 1000)
    assert e.value.status == lib.UNSUPPORTED_TILE
    with pytest.raises(cuda.CtbError) as e:
        cuda.layernorm.layer_norm_fwd(X, v[:100], v, torch.empty_like(X), m, m.clone(), 1e-5, 1024)
    assert e.value.status == lib.BAD_ARG

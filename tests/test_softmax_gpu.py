"""GPU parity of the row-softmax kernels against the float64 oracle.

Tolerance (f32): max|out-ref| / max|ref| <= 1e-5; the reference's own check is
per row atol=1e-5, rtol=1e-4 (examples/softmax.jl:185)."""
import numpy as np
import pytest

from oracle import inputs, ref

pytestmark = pytest.mark.gpu
TOL = 1e-5


def run(cuda, x, variant, tile=None, out=None):
    import torch
    sm = cuda.softmax
    xin = x if isinstance(x, torch.Tensor) else torch.from_numpy(x).cuda()
    out = torch.empty_like(xin) if out is None else out
    N = xin.shape[1]
    if variant == 0:
        sm.softmax_tma_kernel(out, xin, tile or sm.next_power_of_2(N))
    else:
        sm.softmax_chunked_kernel(out, xin, N, tile or 1024)
    torch.cuda.synchronize()
    return out


# the reference's main() cases (examples/softmax.jl:248-256) + ragged and long rows
@pytest.mark.parametrize("M,N", [(256, 256), (1024, 1024), (4096, 4096), (37, 1000), (3, 8192), (1, 4)])
@pytest.mark.parametrize("variant", [0, 1])
def test_softmax_parity(cuda, M, N, variant):
    x = inputs.softmax(M=M, N=N, seed=1)["input"]
    out = run(cuda, x, variant).cpu().numpy()
    want = ref.softmax(x)
    assert ref.max_abs_over_max(out, want) <= TOL
    assert ref.max_rel(out, want) <= 1e-3  # element-wise relative error with the floor 1e-3 * max|ref|
    assert np.abs(out.astype(np.float64).sum(axis=1) - 1).max() < 1e-5
    # the reference's own per-row criterion
    err = np.linalg.norm(out - want, axis=1)
    assert (err <= np.maximum(1e-5, 1e-4 * np.linalg.norm(want, axis=1))).all()


# rows kept in registers, rows kept whole in shared memory (up to 200 KB), rows that are re-read; odd lengths
@pytest.mark.parametrize("M,N", [(5, 333), (2, 20000), (9, 1), (300, 32768), (3, 51200), (2, 60000), (4, 12004)])
def test_softmax_chunked_any_length(cuda, M, N):
    x = inputs.softmax(M=M, N=N, seed=7)["input"]
    out = run(cuda, x, 1).cpu().numpy()
    want = ref.softmax(x)
    assert ref.max_abs_over_max(out, want) <= TOL
    assert ref.max_rel(out, want) <= 1e-3  # element-wise, floored at 1e-3 of the largest probability
    assert np.abs(out.astype(np.float64).sum(axis=1) - 1).max() < 1e-5


def test_softmax_long_f16_rows(cuda):
    x = inputs.softmax(M=5, N=65536, seed=4)["input"].astype(np.float16)  # 128 KB rows: the shared-memory path
    out = run(cuda, x, 1).cpu().numpy()
    assert ref.max_abs_over_max(out, ref.softmax(x)) <= 1e-3


def test_softmax_f16(cuda):
    x = inputs.softmax(M=64, N=2048, seed=3)["input"].astype(np.float16)
    for variant in (0, 1):
        out = run(cuda, x, variant).cpu().numpy()
        assert out.dtype == np.float16
        assert ref.max_abs_over_max(out, ref.softmax(x)) <= 1e-3  # one f16 rounding of the result


def test_softmax_strided_rows_and_extremes(cuda):
    import torch
    x = inputs.softmax(M=16, N=512, seed=2)["input"]
    x[0, :] = -1e30
    x[1, 5] = 1e30
    x[2, :] = 88.0
    big = torch.zeros(16, 640, device="cuda")
    big[:, :512] = torch.from_numpy(x).cuda()
    outbig = torch.full((16, 768), 7.0, device="cuda")
    want = ref.softmax(x)
    for variant in (0, 1):
        run(cuda, big[:, :512], variant, out=outbig[:, :512])
        assert ref.max_abs_over_max(outbig[:, :512].cpu().numpy(), want) <= TOL
        assert (outbig[:, 512:] == 7.0).all()  # nothing written beyond the row


def test_softmax_rejections(cuda):
    import torch
    lib = cuda._lib
    x = torch.zeros(4, 333, device="cuda")
    with pytest.raises(cuda.CtbError) as e:  # rows not 16-byte multiples: single-tile variant refuses
        cuda.softmax.softmax_tma_kernel(torch.empty_like(x), x, 512)
    assert e.value.status == lib.BAD_ALIGN
    x = torch.zeros(4, 1024, device="cuda")
    with pytest.raises(cuda.CtbError) as e:  # tile must be a power of two (src/compiler/intrinsics/core.jl:10-19)
        cuda.softmax.softmax_tma_kernel(torch.empty_like(x), x, 1000)
    assert e.value.status == lib.UNSUPPORTED_TILE
    with pytest.raises(cuda.CtbError) as e:  # tile smaller than the row
        cuda.softmax.softmax_tma_kernel(torch.empty_like(x), x, 512)
    assert e.value.status == lib.UNSUPPORTED_TILE
    x = torch.zeros(2, 16384, device="cuda")
    with pytest.raises(cuda.CtbError) as e:
        cuda.softmax.softmax_tma_kernel(torch.empty_like(x), x, 16384)
    assert e.value.status == lib.UNSUPPORTED
    cuda.softmax.softmax_chunked_kernel(torch.empty(0, 8, device="cuda"), torch.empty(0, 8, device="cuda"), 8, 8)


@pytest.mark.parametrize("M,N", [(3, 1), (700, 127), (5, 128), (2000, 257), (9, 1000), (70, 1024), (70, 1025), (11, 2049),
                                 (600, 4097), (3, 8191), (3, 8193), (400, 16385), (7, 26624), (5, 26625), (310, 50001),
                                 (2, 106497), (3, 212999), (2, 213500)])
@pytest.mark.parametrize("dtype,shift", [(np.float32, 0), (np.float32, 1), (np.float16, 0), (np.float16, 3)])
def test_softmax_any_length_and_alignment(cuda, M, N, dtype, shift):
    """Every kernel and the sizes where one takes over from another: a warp per row, registers of a CTA, one, two, four and
    eight CTAs per row, re-read rows; rows that start anywhere (odd lengths, views off the vector alignment), an output with
    another alignment than the input."""
    import torch
    x = inputs.softmax(M=M, N=N, seed=M + N)["input"].astype(dtype)
    flat = torch.zeros(M * N + 8, device="cuda", dtype=torch.from_numpy(x).dtype)
    flat[shift:shift + M * N] = torch.from_numpy(x).reshape(-1).cuda()
    xin = flat[shift:shift + M * N].view(M, N)
    want = ref.softmax(x)
    for oshift in (shift, 2):
        guard = torch.full((M * N + 8,), 7.0, device="cuda", dtype=xin.dtype)
        out = guard[oshift:oshift + M * N].view(M, N)
        run(cuda, xin, 1, out=out)
        assert ref.max_abs_over_max(out.float().cpu().numpy(), want) <= (TOL if dtype == np.float32 else 1e-3)
        assert (guard[:oshift] == 7.0).all() and (guard[oshift + M * N:] == 7.0).all()
    cuda.check_device_status(0)


@pytest.mark.parametrize("n", [100, 1000, 1001, 1500, 4097, 8192, 9000, 9001, 26003, 60001, 120001, 300001])
@pytest.mark.parametrize("half", [False, True])
def test_softmax_masked_rows(cuda, n, half):
    """Rows with -inf before, behind and between the values, at every alignment, with the type's lowest value, and one that is
    masked as a whole (NaN, as 0 / 0): row kernels of every length give what torch gives in f64."""
    import torch
    dt = torch.float16 if half else torch.float32
    g = torch.Generator(device="cuda").manual_seed(n)
    raw = torch.randn(10 * n + 3, device="cuda", generator=g).to(dt)
    inf = float("inf")
    for off in range(3):
        x = raw.clone()[off:off + 10 * n].view(10, n)
        for r, part in enumerate((slice(0, 1), slice(0, 40), slice(0, n // 2), slice(0, n - 1), slice(n - 1, n), slice(n - 40, n),
                                  slice(1, n))):
            x[r, part] = -inf
        x[7, ::3] = -inf
        x[8, : n // 2] = torch.finfo(dt).min
        x[9] = -inf
        out = torch.full_like(x, 7.0)
        cuda.softmax.softmax_chunked_kernel(out, x, n, 1024)
        want = torch.softmax(x.double(), 1)
        assert out[9].isnan().all() and want[9].isnan().all()
        assert ((out[:9].double() - want[:9]).abs().amax(1) <= (1e-3 if half else 2e-6) * want[:9].amax(1)).all()
        assert (out[:9][x[:9] == -inf] == 0).all()


@pytest.mark.parametrize("M,N,dtype", [(1200, 27001, "float32"), (500, 53003, "float32"), (250, 110001, "float32"), (250, 212001, "float16")])
def test_softmax_clusters_many_rows(cuda, M, N, dtype):
    """Two, four and eight CTAs per row, each with several rows: their two sets of slots and barriers are used again and again, and
    the maximum lies with another CTA in every row."""
    import torch
    g = torch.Generator(device="cuda").manual_seed(N)
    x = torch.randn(M, N, device="cuda", generator=g)
    x[torch.arange(M), (torch.arange(M) * 7919) % N] = 9.0
    x = x.to(getattr(torch, dtype))
    out = torch.empty_like(x)
    for _ in range(2):
        cuda.softmax.softmax_chunked_kernel(out, x, N, 1024)
    want = torch.softmax(x.double(), -1)
    assert ((out - want).abs().amax(1) <= (TOL if dtype == "float32" else 1e-3) * want.amax(1)).all()
    cuda.check_device_status(0)

"""The 32-bit product on tensor cores: every kernel gives a row the same bits, no further from 64 bits than 32-bit additions put it, at the
edges of its tiles; operands that have no three bfloat16 parts come out as plain FMA has them."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def _product(a, w, b=None):
    from qwen25vl_lite.ops import kernels
    out = torch.full((a.shape[0], w.shape[0]), float("nan"), device="cuda")
    kernels.gemm_f32(a, w, b, out, fixed=True)
    assert int(kernels.error_flag(out.device)) == 0
    return out


#  rows, features, K, pitch of the rows beyond K: up to 16 rows a stream; more of them tiles of 32, 64, 96 and 128 rows, with K in parts (where the
#  tiles are few) and whole
CASES = [(1, 15, 256, 0), (2, 33, 288, 0), (3, 3000, 512, 4), (8, 2048, 544, 0), (9, 100, 1056, 0), (16, 16, 11008, 32),
         (17, 127, 256, 0), (33, 129, 288, 0), (64, 2048, 2048, 0), (65, 7000, 320, 4), (97, 9472, 512, 0), (200, 9500, 800, 0), (300, 20000, 256, 12), (1000, 640, 4096, 0),
         # up to four rows, whose lines share their parts: few features, K in one and several spans, a long stream
         (5, 3, 512, 0), (5, 701, 6016, 4), (5, 33, 2080, 0), (17, 2500, 1280, 0), (5, 130, 18944, 0), (5, 9, 33024, 0), (5, 24000, 3072, 0),
         # more than 16 rows: small products as groups of 16 rows, larger ones as tiles of each width
         (50, 300, 1056, 0), (130, 129, 512, 8), (17, 5000, 256, 0), (40, 9000, 288, 0), (90, 20000, 256, 0)]


@pytest.mark.parametrize("m,n,k,extra", CASES)
def test_rows_have_the_same_bits_in_every_kernel(m, n, k, extra):
    gen = torch.Generator(device="cuda").manual_seed(m + n + k)
    a = torch.randn(m, k + extra, generator=gen, device="cuda")[:, :k]
    w, b = torch.randn(n, k, generator=gen, device="cuda"), torch.randn(n, generator=gen, device="cuda")
    out = _product(a, w, b)
    # parts: 2^-24 of the operands' product is left out.  A chunk of 32 k has 12 tensor-core additions, each cut off at 2^-23 of
    # at most the sum of the magnitudes; its value meets up to 7 others in its block, which meets the blocks before, then the bias.
    want, size = a.double() @ w.double().T + b.double(), a.double().abs() @ w.double().abs().T + b.double().abs()
    assert ((out.double() - want).abs() <= (1 + 2 * 12 + 8 + -(-k // 256) + 1) * 2.0 ** -24 * size).all()
    for rows in (1, 2, 4, 7, 16, 17, 50, 130):
        if rows < m:
            assert torch.equal(_product(a[m - rows:], w, b), out[m - rows:]), rows


@pytest.mark.parametrize("m", [5, 60])
def test_rows_that_are_not_aligned(m):
    gen = torch.Generator(device="cuda").manual_seed(m)
    flat, w = torch.randn(m * 513 + 3, generator=gen, device="cuda"), torch.randn(300, 512, generator=gen, device="cuda")
    for first, pitch in ((1, 512), (0, 513)):
        a = flat[first:].as_strided((m, 512), (pitch, 1))
        assert torch.equal(_product(a, w), _product(a.clone(), w))


@pytest.mark.parametrize("m,n", [(3, 260), (16, 260), (40, 260), (40, 9600), (300, 260), (300, 9600)])
def test_operands_without_three_parts(m, n):
    gen = torch.Generator(device="cuda").manual_seed(m)
    a, w = torch.randn(m, 512, generator=gen, device="cuda"), torch.randn(n, 512, generator=gen, device="cuda")
    a[1, 0] = 0.5
    clean = _product(a, w)
    a[m - 1, 7], a[0, 500], w[3, 40], w[259, 0] = float("inf"), float("nan"), float("-inf"), 3.4e38    # the last rounds up to infinity in 16 bits
    want = a.double() @ w.double().T
    want[want.abs() > 3.4028235e38] = want[want.abs() > 3.4028235e38].sign() * float("inf")
    out = _product(a, w)
    assert torch.equal(out.isnan(), want.isnan()) and torch.equal(out.isposinf(), want.isposinf()) and torch.equal(out.isneginf(), want.isneginf())
    assert torch.equal(out[1:m - 1, 4:259], clean[1:m - 1, 4:259])
    assert abs(float(out[1, 259]) / float(want[1, 259]) - 1) < 1e-6


def test_rows_beyond_the_scratch_limit(monkeypatch):
    from qwen25vl_lite.ops import kernels
    gen = torch.Generator(device="cuda").manual_seed(1)
    a, w, b = (torch.randn(*shape, generator=gen, device="cuda") for shape in ((1000, 256), (300, 256), (300,)))
    whole = _product(a, w, b)
    monkeypatch.setattr(kernels, "F32X3_SCRATCH", 1)
    assert torch.equal(_product(a, w, b), whole)


@pytest.mark.parametrize("m,n,k", [(1, 5000, 11008), (16, 5000, 2048), (64, 2048, 11008), (300, 20000, 2048), (300, 2000, 18944)])
def test_rows_that_are_not_numbers(m, n, k):
    """Activations that have all turned into NaN, and rows that hold an infinity: computed again behind the pipeline, so that no wait in it
    runs out, and in a time of the same order."""
    gen = torch.Generator(device="cuda").manual_seed(m)
    a, w = torch.randn(m, k, generator=gen, device="cuda"), torch.randn(n, k, generator=gen, device="cuda")
    out = torch.empty(m, n, device="cuda")
    from qwen25vl_lite.ops import kernels

    def least(x):
        times = []
        for _ in range(4):
            start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            torch.cuda._sleep(200_000)                       # the call is queued before the GPU begins it
            start.record()
            kernels.gemm_f32(x, w, None, out, fixed=True)
            end.record()
            torch.cuda.synchronize()
            times.append(start.elapsed_time(end))
        assert int(kernels.error_flag(out.device)) == 0
        return min(times)

    clean = least(a)
    assert bool(out.isfinite().all())
    whole = out.clone()
    assert least(torch.full_like(a, float("nan"))) < 4 * clean + 0.02
    assert bool(out.isnan().all())
    a[m // 2, k - 1] = float("inf")
    least(a)
    assert torch.equal(out[m // 2], w[:, k - 1].sign() * float("inf"))
    rest = [i for i in range(m) if i != m // 2]
    assert torch.equal(out[rest], whole[rest])


@pytest.mark.parametrize("m,n,k,kernels_of_it", [(16, 300, 512, 1), (40, 300, 512, 1), (300, 20000, 256, 2), (64, 2048, 2048, 3)])
def test_launches_are_counted(m, n, k, kernels_of_it):
    from qwen25vl_lite.ops import kernels
    a, w = torch.randn(m, k, device="cuda"), torch.randn(n, k, device="cuda")
    _product(a, w)
    before = kernels.launch_count()
    kernels.gemm_f32(a, w, None, torch.empty(m, n, device="cuda"))
    assert kernels.launch_count() - before == kernels_of_it


def test_a_second_operand_that_is_not_aligned_takes_no_scratch_memory():
    """It stays with the FMA kernels (in their order), whatever the number of rows."""
    from qwen25vl_lite.ops import kernels
    gen = torch.Generator(device="cuda").manual_seed(3)
    a, flat = torch.randn(3000, 512, generator=gen, device="cuda"), torch.randn(64 * 512 + 1, generator=gen, device="cuda")
    w, out = flat[1:].view(64, 512), torch.empty(3000, 64, device="cuda")
    kernels.gemm_f32(a, w, None, out)
    torch.cuda.synchronize()
    torch.cuda.reset_peak_memory_stats()
    before, launched = torch.cuda.memory_allocated(), kernels.launch_count()
    kernels.gemm_f32(a, w, None, out)
    assert torch.cuda.max_memory_allocated() == before and kernels.launch_count() - launched == 1
    want = a.double() @ w.double().T
    assert float((out.double() - want).norm() / want.norm()) < 3e-7


def _operand(kind, rows, k, gen):
    x = torch.randn(rows, k, generator=gen, device="cuda")
    spread = torch.exp2(torch.rand(rows, k, generator=gen, device="cuda") * 24 - 12)
    return {"both signs": x, "one sign": x.abs(), "spread": x * spread, "spread, one sign": (x * spread).abs(), "very small": x * 2.0 ** -114}[kind]


def _far(out, want):
    return float((out.double() - want).norm() / want.norm())


#  how far from 64 bits a product may be, as a multiple of what the FMA kernels (which take a second operand that is not aligned) are.
#  Measured: both signs 0.54 to 0.66, spread 0.74 to 0.80, one sign up to 1.21 (K 1,024; 0.8 at 11,008), spread with one sign up to 1.84, as the
#  tensor core cuts off where FMA rounds, which sums of one sign collect.  Without one of the six products of parts it would be 15 at least.
KINDS = [("both signs", 1.0), ("spread", 1.0), ("one sign", 1.4), ("spread, one sign", 2.2)]


@pytest.mark.parametrize("kind,factor", KINDS)
@pytest.mark.parametrize("k", [256, 512, 2048, 11008])
def test_error_against_64_bits(kind, factor, k):
    gen = torch.Generator(device="cuda").manual_seed(k)
    a, w = _operand(kind, 300, k, gen), _operand(kind, 1024, k, gen)
    out = _product(a, w)
    want = a.double() @ w.double().T
    shifted = torch.empty(1024 * k + 1, device="cuda")[1:].view(1024, k).copy_(w)
    assert _far(out, want) <= factor * _far(_product(a, shifted), want)
    for rows in (1, 2, 4, 8, 16, 40):                        # the stream of the weights, groups of rows, tiles: the same bits for these operands too
        assert torch.equal(_product(a[:rows], w), out[:rows]), rows


@pytest.mark.parametrize("rows", [1, 3, 7, 16, 50, 300])
def test_every_product_of_parts_counts(rows):
    """Rows in which one place alone is not zero: the result is that product, and exact where it fits 32 bits."""
    parts = 1 + 2.0 ** -9 + 2.0 ** -18                         # three parts: 1, 2^-9, 2^-18
    pairs = [(parts, 2.0), (-0.5, parts), (1 + 2.0 ** -9, 1 + 2.0 ** -9), (2.0 ** -9 + 1, -1 + 2.0 ** -10),
             (parts, 1 + 2.0 ** -5), (1 - 2.0 ** -6, parts)]
    n, k = 257, 288
    for place in (0, 17, 31, 130, 287):
        for x, y in pairs:
            a, w = torch.zeros(rows, k, device="cuda"), torch.zeros(n, k, device="cuda")
            a[:, place], w[:, place] = x, y
            assert bool((_product(a, w) == x * y).all()), (x, y, place)


@pytest.mark.parametrize("m,n", [(1, 300), (4, 300), (16, 300), (60, 300), (64, 2048), (300, 9600)])
def test_very_small_operands_are_taken_whole(m, n):
    gen = torch.Generator(device="cuda").manual_seed(m)
    a, w = _operand("very small", m, 512, gen), torch.randn(n, 512, generator=gen, device="cuda")
    a[0, ::2] = 0
    out, want = _product(a, w), a.double() @ w.double().T
    assert _far(out, want) < 1.5e-7
    assert _far(_product(w[:64], a), want[:, :64].T) < 1.5e-7
    assert torch.equal(_product(torch.zeros_like(a), w), torch.zeros_like(out))

"""The 32-bit product's kernels at the edges of their tiles: a stream of the weights for up to 16 rows, 32 x 32 tiles with the
warps side by side in K, 64 x 64 tiles, and plain loads where TMA refuses an operand.  All add in one order, so a row is the
same bit for bit whichever of them computes it.  (The cases with K 512, 640, 11,008, 544, 4,096 and 384, multiples of 32 from 256 on, run on tensor
cores: test_gemm_f32x3_gpu.py.)"""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

#  rows, features, K, pitch of the rows beyond K
CASES = [(1, 17, 4, 0), (2, 16, 36, 0), (3, 300, 512, 0), (5, 33, 516, 0), (9, 64, 1028, 12), (16, 2400, 640, 0), (4, 16, 11008, 0), (2, 40, 32, 32), (7, 50, 544, 0), (12, 5000, 96, 64),
         (17, 31, 132, 0), (64, 2048, 2052, 0), (33, 65, 4096, 4), (256, 130, 100, 0),                      # warps side by side in K
         (640, 1990, 260, 0), (700, 4100, 128, 8),                                                          # tiles of 64 x 64
         (1, 2400, 224, 0), (2, 17, 192, 32), (3, 300, 224, 0), (4, 16, 96, 0), (7, 50, 160, 0), (8, 2500, 128, 0), (16, 2400, 224, 0),     # the stream: one and two segments
         (33, 65, 4100, 4),                                                                                 # many rounds of warps side by side in K
         (3, 100, 257, 0), (70, 70, 64, 1)]                                                                  # plain loads


@pytest.mark.parametrize("m,n,k,extra", CASES)
def test_gemm_f32_kernels(m, n, k, extra):
    from qwen25vl_lite.ops import kernels
    rng = np.random.default_rng(m + n + k)
    a = torch.tensor(rng.standard_normal((m, k + extra)), dtype=torch.float32, device="cuda")[:, :k]
    w = torch.tensor(rng.standard_normal((n, k)), dtype=torch.float32, device="cuda")
    b = torch.tensor(rng.standard_normal(n), dtype=torch.float32, device="cuda")
    out = torch.full((m, n), float("nan"), device="cuda")
    kernels.gemm_f32(a, w, b, out)
    want = a.double() @ w.double().T + b.double()
    # every product and every addition rounds once: two chains of 64 in a segment, then the segments, then the bias
    steps = 64 + 1 + -(-k // 128) + 1
    bound = steps * 2.0 ** -24 * (a.double().abs() @ w.double().abs().T + b.double().abs()) * 1.01
    assert ((out.double() - want).abs() <= bound).all()
    for rows in (1, 7, 40):                       # the same rows through the kernels for fewer rows
        if rows < m:
            part = torch.empty((rows, n), device="cuda")
            kernels.gemm_f32(a[m - rows:], w, b, part)
            assert torch.equal(part, out[m - rows:])
    strided = torch.full((m, n + 5), 7.0, device="cuda")
    kernels.gemm_f32(a, w, b, strided[:, :n])
    assert torch.equal(strided[:, :n], out) and bool((strided[:, n:] == 7.0).all())
    assert int(kernels.error_flag(out.device)) == 0


@pytest.mark.parametrize("m,n,k,extra", [(9, 100, 16, 0), (16, 24, 12, 4), (4, 32769, 48, 0), (5, 40000, 48, 0), (9, 40000, 64, 0), (16, 33000, 128, 0), (17, 33000, 128, 0),
                                         (2, 33000, 64, 0), (250, 1500, 384, 0), (257, 3000, 132, 0)])
def test_gemm_f32_few_steps_of_k(m, n, k, extra):
    """The sizes at which plain loads and tiles of 64 x 64 take over where K is short."""
    test_gemm_f32_kernels(m, n, k, extra)


@pytest.mark.parametrize("m,n,k", [(1, 30000, 1024), (16, 30000, 1024), (40, 30000, 1024), (40, 2048, 4096), (3, 30000, 1028), (2, 30000, 100)])
def test_gemm_f32_of_a_matrix_just_written(m, n, k):
    """A second operand that the kernel ahead is still writing when this one may begin is waited for, unless the caller says it is fixed."""
    from qwen25vl_lite.ops import kernels
    table = torch.randn(64, k, device="cuda")
    a = torch.randn(m, k, device="cuda")
    for turn in range(4):
        ids = torch.randint(0, 64, (n,), dtype=torch.int32, device="cuda")
        w = torch.full((n, k), float("nan"), device="cuda")
        out, want = torch.empty(m, n, device="cuda"), torch.empty(m, n, device="cuda")
        torch.cuda._sleep(1_000_000)                # both are queued before the first begins
        kernels.embed_gather(table, ids, w)
        kernels.gemm_f32(a, w, None, out)
        torch.cuda.synchronize()
        kernels.gemm_f32(a, w, None, want, fixed=True)
        assert torch.equal(out, want) and not bool(torch.isnan(want).any())

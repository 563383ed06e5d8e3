"""The row-streaming GEMM, the transposing weight-gradient kernel and the fused
bias gradients at the edges of their tiles, against FP64 products of the same
BF16 operands.  FP32 sums of n products of unit-variance operands: within
4 sqrt(n) 2^-24 of the exact sum's scale, 1e-5 of the largest result at the
sizes here; BF16 outputs within 2^-8."""
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.fixture(scope="module")
def nn():
    from finflo_b200 import nn
    nn.build()
    return nn


def _bf(gen, *shape):
    return torch.randn(*shape, generator=gen, device="cuda").to(torch.bfloat16)


def _close(got, ref, tol):
    assert torch.isfinite(got).all()
    assert (got.double() - ref).abs().max() <= tol * ref.abs().max() + 1e-30


@pytest.mark.parametrize("M,N,K", [(4096, 32, 32), (4097, 256, 32), (5000, 16, 32), (4223, 32, 256), (70001, 48, 64), (4300, 20, 16)])
@pytest.mark.parametrize("act", [0, 1])
def test_row_gemm(nn, M, N, K, act):
    gen = torch.Generator(device="cuda").manual_seed(M + N)
    a, b, bias = _bf(gen, M, K), _bf(gen, N, K), torch.randn(N, generator=gen, device="cuda")
    z = torch.zeros(M, N, device="cuda")
    y = torch.zeros(M, N, device="cuda", dtype=torch.bfloat16)
    nn.gemm(a, b, bias=bias, act=act, zf=z, yb=y)
    ref = a.double() @ b.double().T + bias.double()
    _close(z, ref, 1e-5)
    _close(y.float(), torch.nn.functional.silu(ref) if act else ref, 2 ** -8)
    z2 = torch.full((M, N + 4), -7.0, device="cuda")   # a wider row is left alone past N
    nn.gemm(a, b, zf=z2)
    _close(z2[:, :N], ref - bias.double(), 1e-5)
    assert (z2[:, N:] == -7.0).all()
    nn.error()


@pytest.mark.parametrize("M,N,K", [(4096, 256, 256), (4100, 228, 256), (4096, 224, 256), (9344, 256, 256), (9345, 256, 256)])
def test_row_gemm_past_the_shared_memory_of_the_row_kernel(nn, M, N, K):
    """B and one A tile of 256 x 256 take 210 KB, more than the row kernel is
    given: the tile kernel runs, in 32 columns a CTA up to 73 row tiles (9344
    rows), in 256 from there on.  224 columns are the row kernel's last."""
    gen = torch.Generator(device="cuda").manual_seed(M + N)
    a, b = _bf(gen, M, K), _bf(gen, N, K)
    z = torch.full((M, N), -7.0, device="cuda")
    nn.gemm(a, b, zf=z)
    _close(z, a.double() @ b.double().T, 1e-5)
    nn.error()


@pytest.mark.parametrize("rows,N,K", [(1, 8, 8), (16, 512, 256), (63, 32, 32), (64, 16, 32), (65, 256, 32), (1000, 136, 40),
                                      (100003, 32, 32)])
def test_weight_gradient(nn, rows, N, K):
    gen = torch.Generator(device="cuda").manual_seed(rows)
    x, y = _bf(gen, rows, N), _bf(gen, rows, K)
    g = torch.ones(N, K, device="cuda")
    nn.wgrad(x, y, g)
    _close(g, x.double().T @ y.double() + 1.0, 1e-5)
    nn.error()


@pytest.mark.parametrize("rows,cols", [(1, 4), (16, 64), (1000, 32), (4099, 256), (33, 16)])
def test_fused_bias_gradients(nn, rows, cols):
    gen = torch.Generator(device="cuda").manual_seed(rows + cols)
    dy, z = (torch.randn(rows, cols, generator=gen, device="cuda") for _ in range(2))
    dzb = torch.empty(rows, cols, device="cuda", dtype=torch.bfloat16)
    dzf, gb = torch.empty(rows, cols, device="cuda"), torch.zeros(cols, device="cuda")
    nn.silu_bwd_bias(dy, z, dzb, gb, dzf=dzf)
    s = torch.sigmoid(z.double())
    ref = dy.double() * s * (1 + z.double() * (1 - s))
    _close(dzf, ref, 1e-6)
    _close(dzb.float(), ref, 2 ** -8)
    _close(gb, ref.sum(0), 1e-4 if rows > 1 else 1e-6)   # column sums cancel: FP32 of sum |dz| over the sum
    tgt = torch.randn(rows, max(1, cols - 3), generator=gen, device="cuda")
    loss, gb = torch.zeros(1, device="cuda"), torch.zeros(cols, device="cuda")
    nn.mse_bias(z, tgt, dzb, loss, gb, gradf=dzf)
    d = torch.zeros(rows, cols, device="cuda", dtype=torch.float64)
    d[:, :tgt.shape[1]] = z[:, :tgt.shape[1]].double() - tgt.double()
    _close(dzf, 2 * d / tgt.numel(), 1e-6)
    _close(gb, (2 * d / tgt.numel()).sum(0), 1e-4)
    _close(loss, (d * d).sum().reshape(1) / tgt.numel(), 1e-5)

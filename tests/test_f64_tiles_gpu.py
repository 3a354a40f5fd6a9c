"""The f64 tensor-core kernel at the edges of its tiles: both tiles, every K split, both layouts of both
operands, remainders in every dim, views that start anywhere, strides other than 1, a fused addend
and a strided C.  Gate: K roundings of 2^-53 of the sum of absolute products."""
import numpy as np
import pytest
import torch

from gpu_util import dev, host

pytestmark = pytest.mark.gpu


@pytest.fixture
def options(ttb, reset_options):
    yield ttb
    ttb.set_option("mma_tile", -1)
    ttb.set_option("mma_splits", 0)


def _view(rng, shape, form):
    """A device view of `shape`: as is, transposed, starting one element in, or every other element."""
    B, r, c = shape
    a = rng.standard_normal(shape)
    if form == "t":
        return a, dev(a.transpose(0, 2, 1)).permute(0, 2, 1)
    if form == "offset":
        base = torch.zeros(B * r * c + 1, device="cuda", dtype=torch.float64)
        base[1:].copy_(dev(a).reshape(-1))
        return a, base[1:].view(shape)
    if form == "gaps":
        base = torch.zeros((B, r, 2 * c), device="cuda", dtype=torch.float64)
        base[:, :, ::2] = dev(a)
        return a, base[:, :, ::2]
    return a, dev(a)


def _close(got, a, b, add=0.0):
    want = np.matmul(a, b) + add
    bound = (a.shape[2] + 4) * 2.0 ** -53 * (np.matmul(np.abs(a), np.abs(b)) + np.abs(add))
    return (np.abs(got - want) <= 2 * bound).all()  # both sides round


@pytest.mark.parametrize("tile", [0, 1])
@pytest.mark.parametrize("splits", [1, 2, 8])
@pytest.mark.parametrize("shape", [(1, 1, 1, 1), (2, 33, 31, 17), (1, 65, 290, 63), (3, 31, 17, 129), (1, 64, 256, 64)])
def test_tiles_splits_views(options, tile, splits, shape):
    rng = np.random.default_rng(201)
    B, N, K, M = shape
    options.set_option("force_variant", int(options.Variant.DMMA_F64))
    options.set_option("mma_tile", tile)
    options.set_option("mma_splits", splits)
    for fa in ("n", "t", "offset", "gaps"):
        for fb in ("n", "t", "offset", "gaps"):
            a, A = _view(rng, (B, N, K), fa)
            b, Bm = _view(rng, (B, K, M), fb)
            assert _close(host(options.batched_matmul(A, Bm)), a, b), (fa, fb)


@pytest.mark.parametrize("splits", [1, 4])
def test_addend_relu_and_strided_result(options, splits):
    rng = np.random.default_rng(202)
    B, N, K, M = 2, 45, 130, 51
    options.set_option("force_variant", int(options.Variant.DMMA_F64))
    options.set_option("mma_splits", splits)
    a, b = rng.standard_normal((B, N, K)), rng.standard_normal((B, K, M))
    for add in (rng.standard_normal(M), rng.standard_normal((N, 1)), rng.standard_normal((B, N, M))):
        got = host(options.batched_matmul_fused(dev(a), dev(b), dev(add), options.Activation.NONE))
        assert _close(got, a, b, np.broadcast_to(add, (B, N, M)))
        relu = host(options.batched_matmul_fused(dev(a), dev(b), dev(add), options.Activation.RELU))
        assert np.array_equal(relu, np.maximum(got, 0))
    wide = torch.full((B, N, M + 3), 7.0, device="cuda", dtype=torch.float64)
    options.batched_matmul(dev(a), dev(b), out=wide[:, :, 1:M + 1])
    assert _close(host(wide[:, :, 1:M + 1]), a, b)
    assert (wide[:, :, 0] == 7).all() and (wide[:, :, M + 1:] == 7).all()

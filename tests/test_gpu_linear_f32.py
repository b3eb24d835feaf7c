"""The f32 matrix product of the layer-stack executor (csrc/linear_f32.cu) on given inputs: it is called below the C ABI, since
every linear site of a model has a norm in front of it that keeps its inputs near 1."""
import ctypes

import numpy as np
import pytest

from lfm25_inference_b200 import _abi

pytestmark = pytest.mark.gpu

# lfm25::launch_linear_f32(cudaStream_t, const void* x, const void* weight, void* y, size_t m, size_t n, size_t k)
SYMBOL = "_ZN5lfm2517launch_linear_f32EP11CUstream_stPKvS3_Pvmmm"
# row counts of every tile size (16, 32, 64, 96), whole and cut, sums in one CTA and shared by a cluster, sizes that end inside a
# block of 64 of k and inside a tile of 128 columns
SHAPES = [(1, 8, 5), (16, 40, 128), (17, 1000, 130), (33, 1024, 64), (70, 1024, 260), (97, 136, 40), (250, 7168, 129)]


def product(device, x, weight):
    """x [m, k] f32, weight [n, k] of bf16 values."""
    import torch
    launch = getattr(_abi.library(), SYMBOL)
    launch.argtypes = [ctypes.c_void_p] * 4 + [ctypes.c_size_t] * 3
    x = torch.from_numpy(np.ascontiguousarray(x, np.float32)).to(device)
    weight = torch.from_numpy(np.asarray(weight, np.float32)).to(device, torch.bfloat16)
    y = torch.full((x.shape[0], weight.shape[0]), 7.0, device=device)
    stream = torch.cuda.current_stream()
    assert launch(stream.cuda_stream, x.data_ptr(), weight.data_ptr(), y.data_ptr(), *y.shape, x.shape[1]) == 0
    stream.synchronize()
    return y.cpu().numpy()


def sum_bound(k):
    """Part of the sum of the products' sizes that an error may be, with 64 products in a short sum: a rounding (2^-24) for each
    of them, for every pair of them and in a cluster's sum; 2^-21 for what the tensor core cuts on the way (four steps of 16
    products, each of which leaves off less than 2^-23 of the sizes that it adds up: one bit of f32 for the largest of them); and
    2^-23 per 16 products for the two lower parts, which are at most 2^-7 of the first.  Errors measured over these tests' shapes
    and seeds are at most a third of it."""
    return (k / 64 + k / 128 + 8) * 2.0 ** -24 + 2.0 ** -21 + k / 8 * 2.0 ** -30


def spread(rng, shape):
    """f32 values with all 24 bits in use and exponents from -60 to 60 beside one another."""
    values = rng.standard_normal(shape) * 2.0 ** rng.integers(-60, 61, size=shape)
    return values.astype(np.float32)


@pytest.mark.parametrize("m,k,n", SHAPES)
def test_nothing_of_x_is_lost(device, m, k, n):
    """Columns that pick one value of x and scale it by a power of two give it back bit for bit."""
    rng = np.random.default_rng(m)
    x = spread(rng, (m, k))
    picked, scale = rng.integers(0, k, n), 2.0 ** rng.integers(-20, 21, n) * rng.choice([-1.0, 1.0], n)
    weight = np.zeros((n, k))
    weight[np.arange(n), picked] = scale
    assert np.array_equal(product(device, x, weight), (x[:, picked].astype(np.float64) * scale).astype(np.float32))


@pytest.mark.parametrize("m,k,n", SHAPES)
def test_sums(device, m, k, n):
    """Against float64, as part of the sum of the products' sizes."""
    rng = np.random.default_rng(k + m)
    weight = rng.standard_normal((n, k)).astype(np.float32).view(np.uint32) & 0xFFFF0000
    weight = weight.view(np.float32).astype(np.float64)
    for x in (spread(rng, (m, k)), rng.standard_normal((m, k)).astype(np.float32)):
        error = np.abs(product(device, x, weight) - x.astype(np.float64) @ weight.T)
        assert (error <= sum_bound(k) * (np.abs(x).astype(np.float64) @ np.abs(weight).T)).all()


@pytest.mark.parametrize("m,k,n", SHAPES)
def test_values_that_are_no_finite_numbers(device, m, k, n):
    """Infinities and NaN in x, in the weights and in both, zeros against infinities: what the sum of the products is."""
    rng = np.random.default_rng(n)
    odd = np.array([np.inf, -np.inf, np.nan, 0.0])
    x, weight = rng.standard_normal((m, k)).astype(np.float32), rng.choice([-1.5, 0.75, 2.0], size=(n, k))
    for row in range(1, m, 2):
        x[row, rng.integers(0, k)] = odd[row // 2 % 4]
    for row in range(0, n, 3):
        weight[row, rng.integers(0, k)] = odd[row // 3 % 4]
    x[0, 0], weight[0, 0] = 0.0, np.inf
    with np.errstate(invalid="ignore"):
        want = (x.astype(np.float64)[:, None, :] * weight[None]).sum(-1) if m * n * k < 1 << 24 else \
            np.stack([(x.astype(np.float64) * row).sum(-1) for row in weight], 1)
    got = product(device, x, weight)
    assert np.array_equal(np.isnan(got), np.isnan(want))
    infinite = np.isinf(want)
    assert np.array_equal(np.isinf(got), infinite) and np.array_equal(got[infinite], want[infinite].astype(np.float32))
    finite = np.isfinite(want)
    assert finite.any() and np.allclose(got[finite], want[finite], rtol=0, atol=1e-5 * np.sqrt(k))


@pytest.mark.parametrize("m,k,n", [(31, 64, 127), (32, 72, 128), (64, 192, 129), (65, 128, 1), (96, 328, 300), (97, 520, 24),
                                   (400, 2056, 700), (3, 2048, 1100), (16, 2056, 300)])
def test_edges_of_tiles(device, m, k, n):
    """Tiles of 16, 32, 64 and 96 rows by 128 columns, whole and cut; odd and even numbers of 64-wide blocks of k, the last one cut;
    sums in one CTA and in clusters."""
    rng = np.random.default_rng(m * k + n)
    weight = rng.standard_normal((n, k)).astype(np.float32).view(np.uint32) & 0xFFFF0000
    weight = weight.view(np.float32).astype(np.float64)
    for x in (spread(rng, (m, k)), rng.standard_normal((m, k)).astype(np.float32)):
        error = np.abs(product(device, x, weight) - x.astype(np.float64) @ weight.T)
        assert (error <= sum_bound(k) * (np.abs(x).astype(np.float64) @ np.abs(weight).T)).all()

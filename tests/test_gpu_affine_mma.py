"""The affine-grouped linear on the tensor cores (activations as three bf16 parts) against the oracle and 64-bit sums."""
import numpy as np
import pytest

import oracle
import vyre_b200 as vb

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev():
    d = vb.Device.acquire(0)
    yield d
    d.release()


def make(k, n, g, b, seed, dyadic):
    rng = np.random.default_rng(seed)
    w = rng.integers(0, 2**32, size=(k // 8) * n, dtype=np.uint32)
    z = rng.integers(0, 16, size=(k // g) * n, dtype=np.uint32)
    if dyadic:
        return (rng.integers(0, 19, size=b * k).astype(np.float32), w, np.array([0.25, 0.5, 1, 2], np.float32)[rng.integers(0, 4, size=(k // g) * n)], z,
                rng.integers(0, 8, size=n).astype(np.float32))
    # activations of widely different size: 24 significant bits must survive the split
    x = (rng.standard_normal(b * k) * np.exp2(rng.integers(-12, 13, size=b * k))).astype(np.float32)
    return x, w, rng.uniform(1e-3, 2e-2, size=(k // g) * n).astype(np.float32), z, rng.standard_normal(n).astype(np.float32)


def run(dev, args, k, n, g, b):
    prog = (vb.linear_4bit_affine_grouped("x", "w", "s", "z", "b", "o", k, n, g) if b == 1
            else vb.linear_4bit_affine_grouped_batched("x", "w", "s", "z", "b", "o", k, n, g, b))
    sess = vb.ArtifactSession.compile(prog, dev)
    assert sess.kernel_variant() == 5
    return np.frombuffer(sess.run_host(list(args))[0], np.float32).reshape(b, n)


# every column class (2, 5, 8 rows a block; many rows), one and several k chunks, more warps than groups, tails in n and batch
SHAPES = [(4096, 4100, 128, 1), (8192, 2052, 64, 2), (4096, 1372, 32, 3), (2048, 1644, 512, 5), (1536, 1824, 96, 6), (4096, 516, 128, 16), (256, 4096, 64, 33),
          (2816, 100, 352, 61)]


@pytest.mark.parametrize("shape", SHAPES)
def test_tensor_core_sums(dev, shape):
    k, n, g, b = shape
    args = make(k, n, g, b, k + n + b, True)
    assert np.array_equal(run(dev, args, *shape).reshape(-1), oracle.linear_4bit_affine_grouped(*args, k, n, g, batch=b).reshape(-1))
    x, w, s, z, bias = args = make(k, n, g, b, k + n + b + 1, False)
    q = ((w.reshape(k // 8, 1, n) >> (4 * np.arange(8, dtype=np.uint32))[None, :, None]) & 15).reshape(k, n).astype(np.float64)
    wd = (q - np.repeat(z.reshape(-1, n), g, axis=0)) * np.repeat(s.reshape(-1, n).astype(np.float64), g, axis=0)
    xd = x.reshape(b, k).astype(np.float64)
    want = xd @ wd + bias
    # f32 sums of products with |q - 8| <= 8 and a correction with |zp - 8| <= 8, in any order
    mags = np.abs(xd) @ np.repeat(16.0 * s.reshape(-1, n).astype(np.float64), g, axis=0) + np.abs(bias)
    got = run(dev, args, *shape)
    assert np.all(np.abs(got - want) <= (g + k // g + 8) * 2.0 ** -24 * mags)


# several output tiles per block (the next tile's words are fetched under this one's stores, the reduction buffer is used again), with one
# and with several k chunks: up to two rows, sixteen rows a block, eight rows a block with two k slices
@pytest.mark.parametrize("shape", [(512, 40000, 32, 1), (8192, 28676, 128, 1), (256, 20000, 64, 60), (1024, 19300, 32, 50), (256, 12900, 64, 20), (2048, 12804, 64, 17)])
def test_blocks_that_walk_several_tiles(dev, shape):
    test_tensor_core_sums(dev, shape)


# outputs that are no multiple of four: the f32 kernels, whole rows in shared memory up to four batch rows
@pytest.mark.parametrize("shape", [(4096, 4098, 128, 1), (4096, 4098, 64, 1), (4096, 2050, 128, 2), (4096, 2050, 64, 2), (4096, 2050, 128, 3), (4096, 1026, 64, 4),
                                   (4096, 1026, 128, 9)])
def test_other_output_counts_take_the_f32_kernels(dev, shape):
    test_tensor_core_sums(dev, shape)


def definition(x, w, s, z, bias, k, n, g, b):
    """The sums in 64 bits, and the summed magnitudes of their terms."""
    q = ((w.reshape(k // 8, 1, n) >> (4 * np.arange(8, dtype=np.uint32))[None, :, None]) & 15).reshape(k, n).astype(np.float64)
    rep = lambda v: np.repeat(v.reshape(-1, n).astype(np.float64), g, axis=0)  # noqa: E731
    wd, xd = (q - rep(z)) * rep(s), x.reshape(b, k).astype(np.float64)
    return xd @ wd + bias, np.abs(xd) @ (16.0 * rep(s)) + np.abs(bias)


@pytest.mark.parametrize("shape", [(4096, 4096, 128, 1), (1024, 4096, 64, 6), (1024, 4096, 128, 33)])
def test_group_sums_that_overflow_follow_the_definition(dev, shape):
    """Finite activations whose group sums, which meet their scale late, overflow where every scaled weight times x is finite."""
    k, n, g, b = shape
    x, w, s, z, bias = make(k, n, g, b, 11, False)
    x = np.random.default_rng(5).standard_normal(b * k).astype(np.float32)
    w[:] = 0xFFFFFFFF
    z[:] = 1  # every weight is 14 s
    s[:] = np.float32(1e-3)
    x[:k] = 0
    x[[0, 1, 2, g + 3]] = 1e38, 7e37, -9e37, 5e37
    want, mags = definition(x, w, s, z, bias, *shape)
    assert np.all(np.isfinite(want.astype(np.float32)))
    got = run(dev, (x, w, s, z, bias), *shape)
    assert np.all(np.abs(got - want) <= (g + k // g + 8) * 2.0 ** -24 * mags)


def test_scales_whose_zero_point_product_overflows_follow_the_definition(dev):
    k, n, g, b = 1024, 4096, 64, 6
    x, w, s, z, bias = make(k, n, g, b, 12, False)
    x = np.abs(x) * np.float32(1e-12)
    at = 3 * n + np.array([5, 4095])
    s[at], z[at] = 1e30, 2 ** 31  # the weights of that group are -infinity
    got, want = run(dev, (x, w, s, z, bias), k, n, g, b), oracle.linear_4bit_affine_grouped(x, w, s, z, bias, k, n, g, batch=b).reshape(b, n)
    assert np.all(np.isneginf(want[:, [5, 4095]])) and np.array_equal(np.isneginf(got), np.isneginf(want))


@pytest.mark.parametrize("shape", [(4096, 4096, 128, 1), (1024, 4096, 64, 6), (1024, 4096, 128, 33)])
@pytest.mark.parametrize("size", [1e-31, 1e-33, 3e-35])
def test_small_activations_keep_their_bits(dev, shape, size):
    """The residuals of the split become subnormal here; flushed, sixteen bits of an activation or fewer would be left."""
    k, n, g, b = shape
    x, w, s, z, bias = make(k, n, g, b, 13, False)
    rng = np.random.default_rng(6)
    x = np.zeros((b, k), np.float32)
    x[np.arange(b), rng.integers(0, k, size=b)] = rng.uniform(1.0, 2.0, size=b) * size  # one term a sum: no other rounding hides its bits
    s, bias = s * np.float32(4096.0), np.zeros_like(bias)
    want, mags = definition(x, w, s, z, bias, *shape)
    got = run(dev, (x.reshape(-1), w, s, z, bias), *shape)
    # a handful of roundings, and what the split leaves: 2^-133 of an activation, times its weight (|q - zp| <= 15)
    assert np.all(np.abs(got - want) <= 8 * 2.0 ** -24 * mags + 2.0 ** -133 * 15.0 * float(s.max()))


def test_values_that_do_not_split_follow_the_definition(dev):
    k, n, g, b = 1024, 4096, 128, 6
    x, w, s, z, bias = make(k, n, g, b, 3, True)
    w[:] = 0x99999999
    z[:] = 3  # every dequantised weight is 6 s, exactly
    x[2 * k + 5], x[4 * k + 9] = np.inf, np.float32(3.4e38)
    got = run(dev, (x, w, s, z, bias), k, n, g, b)
    assert np.all(np.isposinf(got[2]))
    assert not np.any(np.isnan(got)) and np.all(np.isfinite(got[[0, 1, 3, 5]]))
    want = oracle.linear_4bit_affine_grouped(x, w, s, z, bias, k, n, g, batch=b).reshape(b, n)
    assert np.array_equal(got[[0, 1, 3, 5]], want[[0, 1, 3, 5]])

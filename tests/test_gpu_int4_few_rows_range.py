"""int4 linears of few rows over the whole range of their operands: group sums that f32 does not hold although the outputs are of ordinary size,
scales near its end, infinities and NaN."""
import numpy as np
import pytest

import vyre_b200 as vb
from vyre_b200 import ffi, synth

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def bits(v):
    """float32 values that bf16 holds -> their bits."""
    b = np.ascontiguousarray(v, np.float32).view(np.uint32)
    assert not (b & 0xFFFF).any()
    return (b >> 16).astype(np.uint16)


def run(x, w, s, m, n, k, group, dt):
    d = vb.Device.acquire(0)
    sess = vb.ArtifactSession.compile(vb.linear_int4_grouped_rowmajor("x", "w", "s", "o", m, k, n, group, dt), d)
    out = sess.run_host([x, w.reshape(-1).view(np.uint32), s])[0]
    del sess
    d.release()
    return (np.frombuffer(out, np.float32) if dt == ffi.DT_F32 else synth.bf16_bits_to_f32(np.frombuffer(out, np.uint16))).reshape(m, n)


def definition(x, w, s, n, k, group):
    q = np.stack((w & 15, w >> 4), -1).reshape(n, k).astype(np.float64) - 8.0
    return synth.bf16_bits_to_f32(x).astype(np.float64) @ (q * np.repeat(synth.bf16_bits_to_f32(s).reshape(n, -1).astype(np.float64), group, 1)).T


# one CTA for the whole row and k split over a cluster, both group sizes, a last tile of few outputs, sixteen rows
SHAPES = [(8, 19200, 192, 64), (3, 130, 1600, 64), (5, 300, 1152, 128), (2, 19300, 640, 128), (16, 300, 2048, 128)]


@pytest.mark.parametrize("m,n,k,group", SHAPES)
@pytest.mark.parametrize("what", ["activations", "scales"])
@pytest.mark.parametrize("dt", [ffi.DT_BF16, ffi.DT_F32])
def test_ordinary_outputs_of_extreme_operands(m, n, k, group, what, dt):
    rng = np.random.default_rng(n + k)
    w = rng.integers(0, 256, (n, k // 2), dtype=np.uint8) | 0x88  # q - 8 >= 0: sums grow with every term
    size, step = (2.0**126, 2.0**-110) if what == "activations" else (2.0**-115, 2.0**123)
    x = bits((rng.integers(128, 256, (m, k)) * np.where(rng.random((m, k)) < 0.9, 1.0, -1.0) * (size / 128)).astype(np.float32))
    s = bits((rng.integers(128, 256, (n, k // group)) * (step / 128)).astype(np.float32))
    want, got = definition(x, w, s, n, k, group), run(x, w, s, m, n, k, group, dt)
    assert np.isfinite(want).all() and np.abs(want).max() < 3e38 and np.isfinite(got).all()
    assert (np.abs(got - want) <= (1e-2 if dt == ffi.DT_BF16 else 1e-4) * np.maximum(np.abs(want), 0.1 * np.sqrt(np.mean(want**2)))).all()


@pytest.mark.parametrize("m,n,k,group", SHAPES[:4])
def test_infinities_and_nan(m, n, k, group):
    x, w, s = synth.int4_linear_inputs(m, n, k, group=group, seed=n)
    x, s = x.reshape(m, k).copy(), s.copy()
    x[m - 1, k - 3] = 0x7F80  # +inf
    s[-1] = 0x7FC1            # NaN: the last output
    with np.errstate(invalid="ignore"):
        want = definition(x, w, s, n, k, group)
    got = run(x, w, s, m, n, k, group, ffi.DT_BF16)
    assert (np.isnan(got) == np.isnan(want)).all() and np.isnan(got[:, n - 1]).all()
    inf = np.isinf(want)
    assert inf[m - 1].any() and not inf[: m - 1].any() and (got[inf] == want[inf]).all()
    fine = np.isfinite(want)
    assert (np.abs(got[fine] - want[fine]) <= 1e-2 * np.maximum(np.abs(want[fine]), 0.1 * np.sqrt(np.mean(want[fine] ** 2)))).all()

"""The batched sines and cosines of the step kernels (scp_b200/csrc/trig.cuh,
vec2.cuh) against extended-precision values: both sides of the branch on large
arguments (pi/4 for sine and cosine, pi/2 for the sine alone), batches of small
angles, of large ones and of both, and the fallback for angles of any size."""
import numpy as np
import pytest

from scp_b200 import native

pytestmark = pytest.mark.gpu

SINCOS, SINCOS_ANY, SINE, PAIR, PAIR_SINE = range(5)


def batch(kind, x):
    x = np.ascontiguousarray(x, dtype=np.float64)
    sn, cs = np.empty_like(x), np.empty_like(x)
    native.check(native.lib().scp_gpu_trig_batch(kind, len(x), x.ctypes.data, sn.ctypes.data, cs.ctypes.data), "trig")
    return sn, cs


def around(v, steps=40):
    """v and its neighbours in double precision and a little further out."""
    near = [v]
    for _ in range(steps):
        near = [np.nextafter(near[0], -np.inf), *near, np.nextafter(near[-1], np.inf)]
    return np.concatenate([near, v + v * np.linspace(-1e-6, 1e-6, 41)])


def angles(limit):
    rng = np.random.default_rng(7)
    edges = np.concatenate([around(k * np.pi / 4) for k in range(1, 17)])
    small = rng.uniform(-np.pi / 4, np.pi / 4, 70000)
    mid = rng.uniform(-4 * np.pi, 4 * np.pi, 70000)
    wide = np.exp(rng.uniform(np.log(1e-8), np.log(limit), 70000)) * rng.choice([-1.0, 1.0], 70000)
    special = np.array([0.0, -0.0, 1e-300, -1e-300, 5e-324, limit * 0.999, -limit * 0.999])
    mixed = np.concatenate([edges, -edges, small[:20000], mid[:20000], wide[:20000], special])
    rng.shuffle(mixed)
    return np.concatenate([small, edges, -edges, mid, wide, mixed])


# Derivation.  u = 2^-53.  Sine and cosine on |r| <= pi/4: the last fused
# operation rounds to u (cosine near 1) or u/2; s = r^2 rounds to u/2 * 0.62 and
# enters with 1/2; the polynomial's own roundings stay below u/4; the two fused
# operations of the reduction round r twice, u/2 each; truncation 8e-18: 2.7 u =
# 3.0e-16.  Sine alone on |r| <= pi/2: r^3 p = r - sin r reaches 0.57 and carries
# three roundings (s, r s, p), 1.7 u; the last operation u/2; the reduction's
# two, u each, times cos r: below 1.1 u where the others are largest; truncation
# 4e-17: 3.7 u = 4.1e-16.  FP32 the same with u = 2^-24 and one more operation in
# the reduction: 2.7 u + u/2 = 1.9e-7.
@pytest.mark.parametrize("kind,limit,tol", [(SINCOS, 2.0 ** 20, 3.0e-16), (SINCOS_ANY, 2.0 ** 20, 3.0e-16),
                                            (SINE, 2.0 ** 20, 4.1e-16), (PAIR, 2.0 ** 12, 1.9e-7),
                                            (PAIR_SINE, 2.0 ** 12, 1.9e-7)])
def test_batches_match_extended_precision(gpu, kind, limit, tol):
    x = angles(limit)
    if kind in (PAIR, PAIR_SINE):
        x = x.astype(np.float32).astype(np.float64)
    sn, cs = batch(kind, x)
    xl = x.astype(np.longdouble)
    assert np.max(np.abs(sn - np.sin(xl))) <= tol
    if kind in (SINCOS, SINCOS_ANY, PAIR):
        assert np.max(np.abs(cs - np.cos(xl))) <= tol


def test_any_size(gpu):
    """Around and far beyond the switch to CUDA's routines at 2^19, alone and
    beside small angles of the same batch."""
    rng = np.random.default_rng(3)
    big = np.concatenate([around(2.0 ** 19), -around(2.0 ** 19),
                          np.exp(rng.uniform(np.log(2.0 ** 18), np.log(1e300), 20000))])
    mixed = np.concatenate([big, rng.uniform(-1, 1, len(big))])
    rng.shuffle(mixed)
    x = np.concatenate([big, mixed])
    sn, cs = batch(SINCOS_ANY, x)
    xl = x.astype(np.longdouble)
    assert np.max(np.abs(sn - np.sin(xl))) <= 3.0e-16
    assert np.max(np.abs(cs - np.cos(xl))) <= 3.0e-16


@pytest.mark.parametrize("kind,width", [(SINCOS, 5), (SINCOS_ANY, 5), (SINE, 7), (PAIR, 10), (PAIR_SINE, 14)])
def test_neighbours_in_a_batch_do_not_matter(gpu, kind, width):
    """An angle's values keep their bits whatever shares its batch, for small
    angles too (with a large one beside them they go through the reduction),
    and what is not finite stays its own."""
    rng = np.random.default_rng(5)
    x = rng.uniform(-0.78, 0.78, 40 * width)
    alone = batch(kind, x)
    y = x.copy()
    y[::width] = rng.uniform(3.0, 12.0, 40)
    y[width * 20::width] = np.nan
    keep = np.arange(len(x)) % width != 0
    if kind in (PAIR, PAIR_SINE):   # both lanes of a pair are compared too
        keep = np.arange(len(x)) % width > 1
    beside = batch(kind, y)
    for a, b in zip(alone, beside):
        assert np.array_equal(a[keep], b[keep])
    assert np.all(np.isnan(beside[0][width * 20::width]))

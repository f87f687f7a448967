"""GPU: what one call of a context leaves for the next.

A context keeps its buffers between calls.  Passes that follow a slab run give what a fresh context
gives; they run the same kernels on the same values, so the results are equal bit for bit.
"""
import numpy as np
import pytest

from cases import random_signals
from elasticisolib_3d_b200 import synthetic as S
from elasticisolib_3d_b200.engine import Propagator, SlabPropagator
from oracle import oracle as O

pytestmark = pytest.mark.gpu

DTW = 0.0005


def _medium(nz, nx, ny):
    el = S.elastic_from_velocity(*S.gaussian_perturbed_model((ny, nx, nz), 2500.0, 1443.0, 2000.0, 0.1, 2.0, 5))
    return O.medium_planes(el, DTW, np.float32)


def _points(rng, nz, nx, ny, n):
    z, x, y = (rng.integers(4, m - 4, size=4 * n) for m in (nz, nx, ny))
    return np.unique((y * nx + x) * nz + z)[:n].astype(np.int64)


def _propagator(nz, nx, ny, nts, sub=4, pad=3, cls=Propagator, **kw):
    return cls(nz, nx, ny, nts, sub, pad, 10.0, 10.0, 10.0, sub * DTW, **kw)


def _equal(a, b):
    for x, y in zip(a, b):
        np.testing.assert_array_equal(x, y)


@pytest.mark.parametrize("first", [False, True])
def test_born_image_after_a_slab_run(first):
    """A slab run leaves its neighbours' planes in the ghost planes of the working levels, which the
    imaging pass's ring of levels takes over (first: the ring exists before the slab run)."""
    nz, nx, ny, nts = 40, 33, 50, 12
    rng = np.random.default_rng(1)
    med = _medium(nz, nx, ny)
    spos = [_points(rng, nz, nx, ny, 4) for _ in range(7)]
    rpos = [_points(rng, nz, nx, ny, 60) for _ in range(7)]
    sl = _propagator(nz, nx, ny, nts, cls=SlabPropagator, devices=(0, 0))
    sl.set_medium(med)
    part, ny0 = sl.slabs[0], sl.sizes[0]
    lspos = [_points(rng, nz, nx, ny0, 4) for _ in range(7)]
    lrpos = [_points(rng, nz, nx, ny0, 60) for _ in range(7)]
    sig, dat = random_signals(lspos, nts, rng), random_signals(lrpos, nts, rng)
    if first:
        part.born_adjoint(sig, dat, lspos, lrpos)
    sl.nl_forward([1e3 * s for s in random_signals(spos, nts, rng)], spos, rpos)
    got = part.born_adjoint(sig, dat, lspos, lrpos)
    fresh = _propagator(nz, nx, ny0, nts)
    fresh.set_medium(med[:, :ny0])
    _equal(got, fresh.born_adjoint(sig, dat, lspos, lrpos))
    fresh.close()
    sl.close()

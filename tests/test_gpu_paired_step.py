"""GPU: the paired stepper's launches over the sizes where they can go wrong, against the FP64 oracle.

The default stepper injects few points and records in its own launch, applies the free surface there,
and runs grids whose rows are no multiple of four cells in padded rows.  The cases cover rows of every
remainder mod 4, odd axes, y runs down to two planes, an odd number of fine steps per sample, sources
and receivers on both sides of the in-launch injection limit (8192 points over the nine components),
records shorter and longer than a replayed group of eight samples, with and without the surface.
The bound is the parity tests' 1e-5 relative L2 (FP32 rounding over the steps).
"""
import numpy as np
import pytest

from cases import random_signals, rel_l2
from elasticisolib_3d_b200 import synthetic as S
from elasticisolib_3d_b200.engine import Propagator
from oracle import oracle as O

pytestmark = pytest.mark.gpu

GRIDS = [(17, 13, 10, 12, 2, 3, 40), (29, 21, 19, 8, 3, 3, 60), (42, 24, 30, 21, 4, 1000, 50),
         (30, 27, 18, 5, 5, 2, 950), (72, 40, 57, 6, 4, 4, 1000)]


def _points(rng, nz, nx, ny, n):
    cells = (nz - 8) * (nx - 8) * (ny - 8)
    c = rng.permutation(cells)[:min(n, cells)]
    z, x, y = c % (nz - 8) + 4, c // (nz - 8) % (nx - 8) + 4, c // ((nz - 8) * (nx - 8)) + 4
    return ((y * nx + x) * nz + z).astype(np.int64)


@pytest.mark.parametrize("surface", [0, 1])
@pytest.mark.parametrize("adjoint", [False, True])
@pytest.mark.parametrize("nz,nx,ny,nts,sub,nsrc,nrec", GRIDS)
def test_paired_step_matches_oracle(nz, nx, ny, nts, sub, nsrc, nrec, adjoint, surface):
    rng = np.random.default_rng(nz + 2 * surface)
    el = S.elastic_from_velocity(*S.gaussian_perturbed_model((ny, nx, nz), 2500.0, 1443.0, 2000.0, 0.1, 2.0, 5))
    dts = 0.0005 * sub
    med = O.medium_planes(el, dts / sub, np.float32)
    p = O.PropParams(nz, nx, ny, nts, sub, 3, 10.0, 10.0, 10.0, dts, free_surface=surface)
    spos = [_points(rng, nz, nx, ny, nsrc) for _ in range(7)]
    rpos = [_points(rng, nz, nx, ny, nrec) for _ in range(7)]
    pr = Propagator(nz, nx, ny, nts, sub, 3, 10.0, 10.0, 10.0, dts, free_surface=surface)
    pr.set_medium(med)
    med64 = med.astype(np.float64)
    for _ in range(2):  # a second call reuses the first one's tables and levels
        sig = random_signals(rpos if adjoint else spos, nts, rng)
        sig64 = [s.astype(np.float64) for s in sig]
        if adjoint:
            got = pr.nl_adjoint(sig, spos, rpos)
            ref = O.nl_adjoint_reg(p, med64, sig64, spos, rpos, np.float64)
        else:
            got = pr.nl_forward(sig, spos, rpos)
            ref = O.nl_forward_reg(p, med64, sig64, spos, rpos, np.float64)
        assert rel_l2(got, ref) < 1e-5
    pr.close()


@pytest.mark.parametrize("nz,nx,ny,nts,sub,nsrc,nrec", GRIDS)
def test_born_pair_matches_oracle(nz, nx, ny, nts, sub, nsrc, nrec):
    """The linearised pair on the same grids: secondary sources in the paired step, source levels
    decimated from a ring, the image in the caller's rows (test_gpu_parity's 1e-5)."""
    rng = np.random.default_rng(nz)
    el = S.elastic_from_velocity(*S.gaussian_perturbed_model((ny, nx, nz), 2500.0, 1443.0, 2000.0, 0.1, 2.0, 5))
    dts = 0.0005 * sub
    med = O.medium_planes(el, dts / sub, np.float32)
    p = O.PropParams(nz, nx, ny, nts, sub, 3, 10.0, 10.0, 10.0, dts)
    spos = [_points(rng, nz, nx, ny, nsrc) for _ in range(7)]
    rpos = [_points(rng, nz, nx, ny, nrec) for _ in range(7)]
    sig, dat = random_signals(spos, nts, rng), random_signals(rpos, nts, rng)
    pert = rng.standard_normal((8, ny, nx, nz)).astype(np.float32)
    pr = Propagator(nz, nx, ny, nts, sub, 3, 10.0, 10.0, 10.0, dts)
    pr.set_medium(med)
    up = [[x.astype(np.float64) for x in a] for a in (sig, dat)]
    got = pr.born_forward(sig, pert, spos, rpos)
    ref = O.born_forward_reg(p, med.astype(np.float64), up[0], pert.astype(np.float64), spos, rpos, np.float64)
    assert rel_l2(got, ref) < 1e-5
    got = pr.born_adjoint(sig, dat, spos, rpos)
    ref = O.born_adjoint_reg(p, med.astype(np.float64), up[0], up[1], spos, rpos, None, np.float64)
    assert rel_l2(got, ref) < 1e-5
    pr.close()


def test_padded_rows_give_way_to_memory():
    """A batch that fits the device in unpadded rows only (72-cell rows: a third more when padded) runs,
    with the traces of one that had the room."""
    import torch
    nz, nx, ny, nts, sub, shots = 72, 200, 200, 4, 4, 10
    rng = np.random.default_rng(3)
    el = S.elastic_from_velocity(*S.gaussian_perturbed_model((ny, nx, nz), 2500.0, 1443.0, 2000.0, 0.1, 2.0, 5))
    med = O.medium_planes(el, 0.0005, np.float32)
    spos = [[_points(rng, nz, nx, ny, 5) for _ in range(7)] for _ in range(shots)]
    rpos = [_points(rng, nz, nx, ny, 300) for _ in range(7)]
    models = [random_signals(sp, nts, rng) for sp in spos]
    out = []
    for full in (False, True):
        pr = Propagator(nz, nx, ny, nts, sub, 8, 10.0, 10.0, 10.0, 0.002, q2compat=0)
        pr.set_medium(med)
        torch.cuda.empty_cache()
        hog = None
        if full:
            free, _ = torch.cuda.mem_get_info()
            hog = torch.empty(int(free - 18 * 4 * nz * nx * ny * shots * 1.15 - (64 << 20)), dtype=torch.uint8,
                              device="cuda")
        out.append(pr.nl_forward_batch(models, spos, rpos))
        pr.close()
        del hog
        torch.cuda.empty_cache()
    for a, b in zip(*out):
        for x, y in zip(a, b):
            np.testing.assert_array_equal(x, y)


ODD = [(29, 21, 19, 8, 3), (45, 24, 31, 6, 4), (31, 20, 26, 7, 2)]
LOADERS = [(8, 2, "plain"), (16, 2, "plain"), (8, 2, "cpasync"), (16, 2, "cpasync"), (8, 3, "cpasync"), (8, 2, "tma"),
           (16, 2, "tma"), (8, 3, "tma"), (8, 2, "tma-ring"), (8, 2, "tma-ring-ldg"), (8, 2, "tma-ring-ldg2"),
           (8, 2, "split"), (8, 3, "split"), (8, 4, "split"), (8, 3, "split-fwd"), (8, 2, "split-pair"),
           (8, 4, "split-pair")]


def _odd_case(nz, nx, ny, nts, sub):
    rng = np.random.default_rng(nz)
    el = S.elastic_from_velocity(*S.gaussian_perturbed_model((ny, nx, nz), 2500.0, 1443.0, 2000.0, 0.1, 2.0, 5))
    dts = 0.0005 * sub
    med = O.medium_planes(el, dts / sub, np.float32)
    p = O.PropParams(nz, nx, ny, nts, sub, 3, 10.0, 10.0, 10.0, dts)
    spos = [_points(rng, nz, nx, ny, 4) for _ in range(7)]
    rpos = [_points(rng, nz, nx, ny, 50) for _ in range(7)]
    pr = Propagator(nz, nx, ny, nts, sub, 3, 10.0, 10.0, 10.0, dts)
    pr.set_medium(med)
    return rng, p, med.astype(np.float64), spos, rpos, pr


@pytest.mark.parametrize("nz,nx,ny,nts,sub", ODD)
def test_every_stepper_on_odd_rows(nz, nx, ny, nts, sub):
    """The stepper forms that once took rows of a multiple of four cells only, on rows that are not."""
    rng, p, med, spos, rpos, pr = _odd_case(nz, nx, ny, nts, sub)
    sig, dat = random_signals(spos, nts, rng), random_signals(rpos, nts, rng)
    fwd = O.nl_forward_reg(p, med, [s.astype(np.float64) for s in sig], spos, rpos, np.float64)
    adj = O.nl_adjoint_reg(p, med, [d.astype(np.float64) for d in dat], spos, rpos, np.float64)
    for v in LOADERS:
        pr.set_stepper_variant(*v)
        assert rel_l2(pr.nl_forward(sig, spos, rpos), fwd) < 1e-5, v
        assert rel_l2(pr.nl_adjoint(dat, spos, rpos), adj) < 1e-5, v
    pr.close()


@pytest.mark.parametrize("nz,nx,ny,nts,sub", ODD)
def test_image_forms_on_odd_rows(nz, nx, ny, nts, sub):
    """The Born adjoint on such rows with every imaging kernel, adjoint state, decimation and storage
    (FP16 states and slots within the 1e-3 that they are allowed on other grids)."""
    rng, p, med, spos, rpos, pr = _odd_case(nz, nx, ny, nts, sub)
    sig, dat = random_signals(spos, nts, rng), random_signals(rpos, nts, rng)
    ref = O.born_adjoint_reg(p, med, [s.astype(np.float64) for s in sig], [d.astype(np.float64) for d in dat], spos,
                             rpos, None, np.float64)

    def check(bound, **how):
        pr.set_stepper_variant(*how.get("variant", (8, 3, "split-pair")))
        pr.set_premultiplied_adjoint(how.get("prem", True))
        pr.set_decimation_ring(how.get("ring", True))
        pr.set_imaging_variant(how.get("imaging", "auto"))
        pr.set_checkpoint_policy(how.get("store", "fp32"), how.get("segment", 3))
        pr.set_velocity_storage(how.get("store", "fp32"))
        assert rel_l2(pr.born_adjoint(sig, dat, spos, rpos), ref) < bound, how

    for imaging in ("cells", "tma", "tma-levels", "tma-levels-4"):
        for prem in (True, False):
            check(1e-5, imaging=imaging, prem=prem)
    for variant in ((8, 2, "plain"), (8, 2, "cpasync"), (8, 2, "tma"), (16, 2, "tma"), (8, 3, "split"),
                    (8, 3, "split-fwd")):
        check(1e-5, variant=variant)
        check(1e-5, variant=variant, ring=False)
    check(1e-5, ring=False)
    check(1e-3, store="fp16", segment=2)
    check(1e-3, store="fp16", segment=2, ring=False)
    pr.close()


def test_autotuner_takes_a_fast_stepper_on_odd_rows():
    """Rows of an odd number of cells run every stepper: the plain one, three times slower than the
    default on such a grid, is not what the autotuner picks."""
    from elasticisolib_3d_b200 import autotune as AT
    nz, nx, ny = 101, 91, 117
    el = S.elastic_from_velocity(*S.gaussian_perturbed_model((ny, nx, nz), 2500.0, 1443.0, 2000.0, 0.1, 2.0, 5))
    pr = Propagator(nz, nx, ny, 10, 4, 8, 10.0, 10.0, 10.0, 0.002)
    pr.set_medium(O.medium_planes(el, 0.0005, np.float32))
    best, times = AT.autotune(pr, mode=0, steps=6, warmup=2)
    assert len(times) == len(AT.CANDIDATES) and best[2] in AT.TMA_LOADERS
    best_g, per = AT.autotune_gradient(pr, steps=4, warmup=1)
    assert best_g[2] in AT.TMA_LOADERS and len(per[best_g]) == 2
    pr.close()

"""Calls that fail after a deposit pass: what the next calls see.  A call that
returns an error leaves no deposited weights behind, so the next gx_masset
gives the particles' mass and nothing on top of it."""
import numpy as np
import pytest

from galaxy_b200 import (Galaxy, GxError, make_config, GX_FLAG_SORTED_DEPOSIT, GX_GRID_MASS, GX_PREC_FP64,
                         GX_PREC_MIXED, GX_RMAP_STDPOL)
from galaxy_b200.disk import exp_disk, kt_disk

pytestmark = pytest.mark.gpu


def cfg2(flags=0, **kw):
    return make_config(2, 40, 64, nsect=1, rmap=GX_RMAP_STDPOL, softl=1.0, tsoft=2, flags=flags, **kw)


def test_refused_adjoint_leaves_the_mass_as_it_was():
    """Every harmonic skipped: the adjoint has no solve to differentiate and
    refuses.  The mass array is the particles' before and after, and masset
    gives it again, bit for bit."""
    rec, pm = kt_disk(5000, seed=2, rmax=4.9, ndim=2, dt=0.05, lscale=10.0)
    with Galaxy(cfg2(ng=3, skip=(0, 1, 2), pmass=pm)) as gal:
        gal.greenm()
        gal.loadup(rec)
        gal.masset()
        mass = gal.grid(GX_GRID_MASS)
        assert mass.sum() > 0
        for _ in range(2):
            with pytest.raises(GxError):
                gal.adjoint(3, 2)
            assert np.array_equal(gal.grid(GX_GRID_MASS), mass)
        with pytest.raises(GxError):
            gal.step(2)
        assert np.array_equal(gal.unload(), rec)
        gal.masset()
        assert np.array_equal(gal.grid(GX_GRID_MASS), mass)
        # without a step there is nothing to solve
        J, grad, _, _ = gal.adjoint(0, 1)
        assert J > 0 and np.isfinite(grad).all()


@pytest.mark.parametrize("flags", [0, GX_FLAG_SORTED_DEPOSIT])
def test_zoned_run_that_fails_leaves_no_deposit_behind(flags):
    """Step factors that are not multiples of one another (1, 4, 6): the
    seventh step finds a zone's older mass array at a useless time and the call
    fails after its particle pass.  The run loaded again starts as a fresh one."""
    rec, pm = kt_disk(20000, seed=5, rmax=4.9, ndim=2, dt=0.05, lscale=10.0)
    with Galaxy(cfg2(flags, ng=9, pmass=pm)) as gal:
        gal.greenm()
        gal.set_zones([1, 4, 6], [0.0, 3.0, 12.0])
        gal.loadup(rec)
        gal.masset()
        mass = gal.grid(GX_GRID_MASS)
        gal.step(3)
        ref = gal.unload(), gal.grid(GX_GRID_MASS)
        with pytest.raises(GxError):
            gal.step(4)
        gal.loadup(rec)
        gal.masset()
        assert np.array_equal(gal.grid(GX_GRID_MASS), mass)
        gal.step(3)
        assert np.array_equal(gal.unload(), ref[0])
        assert np.array_equal(gal.grid(GX_GRID_MASS), ref[1])


def almost_full(left):
    """All of the device's free memory but `left` bytes, held until released"""
    import torch
    torch.cuda.init()
    return torch.empty(torch.cuda.mem_get_info()[0] - left, dtype=torch.uint8, device="cuda")


def release():
    import torch
    torch.cuda.empty_cache()


def test_allocation_that_fails_does_not_fail_the_next_call():
    """A call that finds no memory returns that error, and the next one, with
    memory again, is not told of it."""
    rec, pm = kt_disk(20000, seed=5, rmax=4.9, ndim=2, dt=0.05, lscale=10.0)
    out = []
    for full in (False, True):
        with Galaxy(cfg2(ng=9, pmass=pm)) as gal:
            gal.greenm()
            gal.loadup(rec)
            gal.masset()
            if full:
                hold = almost_full(4 << 20)
                try:
                    with pytest.raises(GxError):
                        gal.greenm()
                finally:
                    del hold
                    release()
            gal.step(2)
            out.append(gal.unload())
    assert np.array_equal(*out)


@pytest.mark.parametrize("precision", [GX_PREC_MIXED, GX_PREC_FP64])
def test_particles_that_do_not_fit_leave_an_empty_context(precision):
    """loadup of more particles than the device holds, in a context that has
    some: afterwards it has none, and takes the old ones again.  The steps are
    those of a fresh context (FP64: up to the order of its atomics)."""
    rec, pm = kt_disk(20000, seed=5, rmax=4.9, ndim=2, dt=0.05, lscale=10.0)
    big = np.zeros((3_000_000, 4), np.float32)  # more than 100 bytes a particle in device arrays
    out = []
    for full in (False, True):
        with Galaxy(cfg2(ng=9, pmass=pm, precision=precision)) as gal:
            gal.greenm()
            gal.loadup(rec)
            gal.masset()
            if full:
                hold = almost_full(100 << 20)
                try:
                    with pytest.raises(GxError):
                        gal.loadup(big)
                    with pytest.raises(GxError):
                        gal.step(1)  # no mass array
                    assert not gal.unload().any()
                    gal.loadup(rec)
                    gal.masset()
                finally:
                    del hold
                    release()
            gal.step(2)
            out.append(gal.unload())
    if precision == GX_PREC_MIXED:
        assert np.array_equal(*out)
    else:
        assert np.abs(out[0] - out[1]).max() <= 1e-6 * np.abs(out[0]).max()


def test_sfp_particles_that_do_not_fit_leave_an_empty_handle(golden_dir):
    import os
    from galaxy_b200.sfp import Basis, Sfp
    basis = Basis.from_json(os.path.join(golden_dir, "aj07.json"), maxm=8, maxn=19)
    pos = exp_disk(20000, seed=4)
    big = np.zeros((3_000_000, 2), np.float32)  # 80 bytes a particle
    with Sfp(basis, 6.0) as s:
        s.load(pos)
        ref = s.sum()
        hold = almost_full(100 << 20)
        try:
            with pytest.raises(GxError):
                s.load(big)
            assert not s.sum().any() and not s.unload().any()
            s.load(pos)
            assert np.array_equal(s.sum(), ref)
        finally:
            del hold
            release()

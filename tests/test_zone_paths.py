"""Time-step zones: the direct path (particles moved in place, their weights
added straight into the zones' accumulators) against the sorted one
(GX_FLAG_SORTED_DEPOSIT: the per-zone counting-sort deposit).  Both add the
same integers and convert them the same way, so zone codes, ring ranges,
masses and records agree bit for bit."""
import numpy as np
import pytest

from galaxy_b200 import (Galaxy, make_config, GX_FLAG_QUADRATIC, GX_FLAG_SORTED_DEPOSIT, GX_GRID_MASS,
                         GX_RMAP_LOG, GX_RMAP_STDPOL)
from galaxy_b200.disk import kt_disk

pytestmark = pytest.mark.gpu


def cfg2(flags):
    return make_config(2, 40, 64, ng=9, nsect=2, rmap=GX_RMAP_STDPOL, softl=1.0, tsoft=2, flags=flags)


def cfg3(flags):
    return make_config(3, 31, 50, ngz=15, dzg=0.1, ng=7, rmap=GX_RMAP_LOG, rmap_a=float(np.log(100.0) / 30),
                       rmap_r0=0.05, softl=0.2, tsoft=1, halo=1, halo_v2=0.49 * 0.025 ** 2, halo_rc=1.0, flags=flags)


@pytest.mark.parametrize("ndim,flags,nstep,zbr,n", [
    (2, 0, [1, 2], [0.0, 12.0], 20011),
    (2, 0, [1, 2, 4], [0.0, 3.0, 12.0], 255),
    (2, 0, [1, 3], [0.0, 12.0], 0),
    (3, 0, [1, 2, 4], [0.0, 0.7, 2.0], 30000),
    (3, GX_FLAG_QUADRATIC, [1, 2], [0.0, 1.0], 9001),
    (2, 0, [1, 2], [0.0, 12.0], 700001),
])
def test_direct_zone_steps_equal_the_sorted_ones(ndim, flags, nstep, zbr, n):
    L = 10.0 if ndim == 2 else 1.0
    rec, pm = kt_disk(max(n, 1), seed=5, rmax=4.9, ndim=ndim, z0=0.1, dt=0.05, lscale=L)
    rec = rec[:n]
    if n:
        rec[::50] *= np.float32(1.7)  # some beyond the grid's edge, some fast
    out = []
    for f in (flags, flags | GX_FLAG_SORTED_DEPOSIT):
        cfg = (cfg2 if ndim == 2 else cfg3)(f)
        cfg.pmass = pm
        with Galaxy(cfg) as gal:
            gal.greenm()
            gal.set_zones(nstep, zbr)
            gal.loadup(rec)
            gal.masset()
            res = [gal.grid(GX_GRID_MASS)]
            for k in (1, 2, 2 * max(nstep)):
                gal.step(k)
                res += [gal.grid(GX_GRID_MASS), gal.unload(), *gal.zone_rings(), *gal.zone_info()]
        out.append(res)
    for a, b in zip(*out):
        assert np.array_equal(a, b)
    if n > 1000:
        assert len(np.unique(out[0][-2])) == len(nstep) + 1  # every zone and the off-grid list


def test_zones_without_room_for_their_accumulators():
    """A large mesh on a nearly full device: the zones' integer accumulators
    (twice their mass arrays) do not fit, and the run takes the sorted path,
    which does without them; the same bits."""
    import torch
    cfg = make_config(2, 4096, 512, ng=1, rmap=GX_RMAP_LOG, rmap_a=float(np.log(100.0) / 4095), rmap_r0=0.05,
                      softl=0.05, tsoft=1)
    rec, pm = kt_disk(30000, seed=6, rmax=4.9, ndim=2, dt=0.05)
    cfg.pmass = pm
    out = []
    for full in (False, True):
        with Galaxy(cfg) as gal:
            hold = None
            if full:
                # mass arrays of three more zones 50 MB, their accumulators 50 MB
                gal.loadup(rec)   # the particle arrays first
                gal.loadup(rec[:0])
                hold = torch.empty(torch.cuda.mem_get_info()[0] - (80 << 20), dtype=torch.uint8, device="cuda")
            try:
                gal.set_zones([1, 2, 4, 8], [0.0, 1.0, 2.0, 3.0])
            finally:
                del hold
                torch.cuda.empty_cache()
            gal.loadup(rec)
            gal.masset()
            out.append((gal.grid(GX_GRID_MASS), *gal.zone_info()[:1]))
    for a, b in zip(*out):
        assert np.array_equal(a, b)

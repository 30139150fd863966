"""The fused particle pass on the bucketed store (gx_bucket.cu) against the
row-sorted deposit (gx_deposit.cu, GX_FLAG_SORTED_DEPOSIT).

Both compute the same positions (the same push arithmetic) and the same
integer fixed-point mass sums, so every case must agree bit for bit: the
particles (read back in load order) and the mass array, after steps that
cross the entry points which compact the bucketed store (getacc, tmcent,
icheck, unload) and re-bucket it.  Cases: 3D and 2D discs; the compensated
position update; particles moving several cells per step (segments
overflow, corners fall outside the deposit window, particles leave the
grid); the 3D benchmark grid; a context with no particles."""
import numpy as np
import pytest

from galaxy_b200 import (Galaxy, make_config, GX_FLAG_COMPENSATED, GX_FLAG_QUADRATIC, GX_FLAG_SORTED_DEPOSIT,
                         GX_RMAP_LOG, GX_RMAP_STDPOL, GX_GRID_MASS)
from galaxy_b200.disk import kt_disk

pytestmark = pytest.mark.gpu


def cfg3(nr=32, na=64, ngz=15, dzg=0.1, ng=9, softl=0.2):
    return make_config(3, nr, na, ngz=ngz, dzg=dzg, ng=ng, rmap=GX_RMAP_LOG,
                       rmap_a=float(np.log(100.0) / (nr - 1)), rmap_r0=0.05, softl=softl, tsoft=1)


def cfg2():
    return make_config(2, 40, 64, ng=9, rmap=GX_RMAP_STDPOL, softl=1.0, tsoft=1)


def case(name):
    if name == "3d":
        rec, pm = kt_disk(200_000, seed=1, rmax=4.5, ndim=3, z0=0.1, dt=0.025)
        return cfg3(), rec, pm, 0
    if name == "2d":
        rec, pm = kt_disk(200_000, seed=2, rmax=5.0, ndim=2, dt=0.025, lscale=5.0)
        return cfg2(), rec, pm, 0
    if name == "3d-compensated":
        rec, pm = kt_disk(100_000, seed=3, rmax=4.5, ndim=3, z0=0.1, dt=0.025)
        return cfg3(), rec, pm, GX_FLAG_COMPENSATED
    if name == "3d-fast-movers":
        rec, pm = kt_disk(100_000, seed=4, rmax=4.5, ndim=3, z0=0.1, dt=0.025)
        rec = rec.copy()
        rec[:, 3:] *= 25.0   # several cells per step: overflow, out-of-window corners, off-grid
        return cfg3(), rec, pm, 0
    if name == "2d-fast-movers":
        rec, pm = kt_disk(100_000, seed=5, rmax=5.0, ndim=2, dt=0.025, lscale=5.0)
        rec = rec.copy()
        rec[:, 2:] *= 25.0
        return cfg2(), rec, pm, 0
    if name.startswith("3d-quadratic"):
        nr, na, ngz = (32, 64, 15) if name == "3d-quadratic" else (29, 50, 27)
        rec, pm = kt_disk(200_000 if name == "3d-quadratic" else 60_000, seed=6, rmax=4.5, ndim=3, z0=0.1, dt=0.025)
        rec = rec.copy()
        rec[::40, 2] *= 6.0    # to the lowest and highest planes, and off the grid
        rec[::30, :2] *= 0.1   # to the clamped inner ring and the hole
        rec[::50, 3:] *= 20.0  # several cells per step
        flags = GX_FLAG_QUADRATIC | (0 if name == "3d-quadratic" else GX_FLAG_COMPENSATED)
        return cfg3(nr=nr, na=na, ngz=ngz), rec, pm, flags
    if name.startswith("wide"):
        # the widest deposit windows and field rows (512 spokes; 444 is the
        # largest fused quadratic grid), with particles for items that stage the
        # rows and with too few for it
        _, na, scheme, n = name.split("-")
        rec, pm = kt_disk(int(n), seed=9, rmax=4.5, ndim=3, z0=0.1, dt=0.025)
        rec = rec.copy()
        rec[::50, 3:] *= 20.0
        flags = {"linear": 0, "compensated": GX_FLAG_COMPENSATED, "quadratic": GX_FLAG_QUADRATIC}[scheme]
        return cfg3(nr=24, na=int(na), ng=5), rec, pm, flags
    if name == "bench3":
        rec, pm = kt_disk(1_000_000, seed=12345, rmax=4.8, ndim=3, z0=0.1, dt=0.02)
        return cfg3(nr=128, na=256, ngz=125, dzg=0.04, ng=17, softl=0.1), rec, pm, 0
    raise KeyError(name)


def run(cfg, rec, pm, flags):
    cfg.pmass = pm
    cfg.flags = flags
    out = []
    with Galaxy(cfg) as gal:
        gal.greenm()
        gal.loadup(rec)
        gal.masset()
        gal.findf(True)
        gal.tmcent(True)
        gal.step(3)
        out.append(gal.grid(GX_GRID_MASS))
        gal.findf(True)
        acc, pot = gal.getacc()        # compacts the bucketed store
        out += [acc, pot]
        gal.step(2)
        gal.findf(True)
        gal.icheck()                   # compacts it again (its sums are not compared)
        gal.step(1, phys=True)
        out.append(gal.unload())
        out.append(gal.grid(GX_GRID_MASS))
        gal.step(2)                    # re-bucketed from the compacted store
        out.append(gal.unload())
        out.append(gal.grid(GX_GRID_MASS))
    return out


@pytest.mark.parametrize("name", ["3d", "2d", "3d-compensated", "3d-fast-movers",
                                  "2d-fast-movers", "bench3", "3d-quadratic",
                                  "3d-quadratic-compensated", "wide-512-linear-150000",
                                  "wide-512-compensated-15000", "wide-444-quadratic-150000",
                                  "wide-444-quadratic-15000", "wide-446-quadratic-15000",
                                  "wide-512-quadratic-15000"])
def test_fused_step_is_bitwise_the_sorted_deposit(name):
    cfg, rec, pm, flags = case(name)
    a = run(cfg, rec, pm, flags)
    b = run(cfg, rec, pm, flags | GX_FLAG_SORTED_DEPOSIT)
    for k, (x, y) in enumerate(zip(a, b)):
        assert x.shape == y.shape
        same = x.view(np.uint32) == y.view(np.uint32)
        assert same.all(), (name, k, int((~same).sum()))
    if "fast" in name:
        # the run did move particles across several rows and off the grid
        pos = a[-2]
        assert np.isfinite(pos).all()


def test_fused_step_empty_context():
    cfg = cfg3()
    cfg.pmass = 1.0
    with Galaxy(cfg) as gal:
        gal.greenm()
        gal.loadup(np.zeros((0, 6), np.float32))
        gal.masset()
        gal.step(2)
        assert gal.unload().shape == (0, 6)
        assert not gal.grid(GX_GRID_MASS).any()


def test_fused_2d_graph_replay_is_bitwise_the_sorted_deposit():
    """A 2D run long enough that the fused path replays pairs of steps from
    a CUDA graph (captured once the mass is a fused pass's): the same
    particles and mass, bit for bit, as the sorted deposit's plain
    launches, over two calls."""
    cfg, rec, pm, _ = case("2d")
    out = []
    for flags in (0, GX_FLAG_SORTED_DEPOSIT):
        cfg.pmass = pm
        cfg.flags = flags
        with Galaxy(cfg) as gal:
            gal.greenm()
            gal.loadup(rec)
            gal.masset()
            gal.step(21)
            gal.step(14, phys=True)
            out.append((gal.unload(), gal.grid(GX_GRID_MASS)))
    for x, y in zip(out[0], out[1]):
        assert (x.view(np.uint32) == y.view(np.uint32)).all()


def lowest_boundary(ngz):
    """dzg and z of a point on the boundary between planes 0 and 1 of the
    quadratic scheme whose plane is 1 by the reference's operations (the
    deposit) and 0 by the multiplication with 1 / dzg (the interpolation)"""
    f = np.float32
    for dzg in np.linspace(0.1, 0.12, 4001).astype(f):
        zm = f(0.5) * dzg * f(ngz - 1)
        z0 = f(0.5) * dzg - zm
        for z in (z0, np.nextafter(z0, f(-9)), np.nextafter(z0, f(9))):
            s = z + zm
            if s * (f(1) / dzg) + f(0.5) < 1 <= s / dzg + f(0.5):
                return float(dzg), z
    raise AssertionError("no such boundary")


def test_fused_quadratic_field_below_the_deposit_planes():
    """Particles that interpolate one plane below their deposit plane, at the
    bottom of the grid: their lowest node lies in the last plane of the ring
    below (flat offsets), which the solve has to cover although no mass is near
    it.  The field there is made non-finite beforehand, so that a plane the
    solve leaves out shows in the particles."""
    ngz = 15
    dzg, z = lowest_boundary(ngz)
    cfg = cfg3(ngz=ngz, dzg=dzg)
    rec, pm = kt_disk(20_000, seed=8, rmax=4.5, ndim=3, z0=0.05, dt=0.025)
    rec = rec[np.abs(rec[:, 2]) < 2 * dzg].copy()  # the planes next to the middle
    rec[:200, 2] = z
    cfg.pmass = pm
    out = []
    for flags in (0, GX_FLAG_SORTED_DEPOSIT):
        cfg.flags = GX_FLAG_QUADRATIC | flags
        with Galaxy(cfg) as gal:
            gal.greenm()
            gal.set_mass(np.full(gal.mesh, 1e38, np.float32))
            gal.findf(True)
            gal.loadup(rec)
            gal.masset()
            gal.step(1)
            out.append(gal.unload())
    assert np.isfinite(out[0]).all()
    assert np.array_equal(out[0].view(np.uint32), out[1].view(np.uint32))

"""The plain FP64 Euler kernel that advances one direction at a time (64 threads per element), which every mesh
of more than 12 elements per SM takes: what the other files try on small meshes, and thereby on the kernel of three
directions at a time, is tried here above that limit -- open boundaries, 2:1 faces with and without blending,
both sets of fluxes, groups with time steps of their own, cooling, a positivity repair that has to act.  Compared
with the oracle bit for bit, as there."""
import numpy as np
import pytest

from nemo_b200 import abi, mesh, setups
from nemo_b200.solver import Solver
from oracle import oracle as orc

pytestmark = pytest.mark.gpu

FLUXES = [(abi.VOLFLUX_CHANDRASHEKAR, abi.SURFFLUX_HLLC), (abi.VOLFLUX_CENTRAL, abi.SURFFLUX_RUSANOV)]


@pytest.fixture(autouse=True)
def _fin():
    yield
    try:
        abi.call("nemo_gpu_finalize")
    except Exception:
        pass


def limit():
    import torch
    return 12 * torch.cuda.get_device_properties(0).multi_processor_count


def box(**kw):
    """A box of at most 156 elements more than the limit."""
    m = mesh.brick(limit() // (12 * 13) + 1, 12, 13, **kw)
    assert m.E > limit()
    return m


def forest():
    m = mesh.forest(8, lambda lvl, c, s: c[:, 1] < 0.5, max_level=1)
    assert m.E > limit() and len(m.mortars()) > 0
    return m


def jumps(m):
    u = setups.smooth_random(m, seed=5)
    u[:, :, 17] *= 1.5   # alpha > 0 in part of the elements
    return u


@pytest.mark.parametrize("blend", [False, True])
@pytest.mark.parametrize("vf,sf", FLUXES)
@pytest.mark.parametrize("make", [lambda: box(periodic=(False,) * 3), forest], ids=["open box", "forest"])
def test_steps_bit_exact(make, vf, sf, blend):
    m = make()
    u = jumps(m)
    c = abi.default_cfg(volume_flux=vf, surface_flux=sf, indicator=abi.IND_MODAL if blend else abi.IND_NONE, positivity=1)
    s = Solver(c, m)
    o = orc.Oracle.for_mesh(c, m)
    s.upload(u)
    assert np.array_equal(s.rhs(), o.rhs(u, alpha=o.alpha(u)) if blend else o.rhs(u))
    t, n = s.run(nsteps=2)
    ref, tr, nr, _ = o.run(u, nsteps=2)
    assert t == tr and n == nr
    assert np.array_equal(s.download(), ref)


def test_groups_bit_exact():
    """Two boxes as groups of one run, each with its own time step: both as the oracle advances them alone."""
    b = mesh.brick(limit() // 144 // 2 + 1, 12, 12)
    us = [setups.gaussian_blob(b, a) for a in (0.1, 1.0)]
    m, g = mesh.concat([b, b])
    assert m.E > limit()
    c = abi.default_cfg(indicator=abi.IND_MODAL, positivity=1)
    s = Solver(c, m, g)
    s.upload(np.concatenate(us, axis=1))
    s.run(nsteps=2)
    got = s.download()
    for i, u in enumerate(us):
        ref, _, _, _ = orc.Oracle.for_mesh(c, b).run(u, nsteps=2)
        assert np.array_equal(got[:, i * b.E: (i + 1) * b.E], ref), i


def test_cooled_run_bit_exact():
    m = box()
    u = setups.smooth_random(m, seed=6, kappa=1.1)
    c = abi.default_cfg(kappa=1.1, indicator=abi.IND_MODAL, positivity=1, source=abi.SOURCE_BAROTROPIC_COOLING,
                        dens_critical=1.0, k_isothermal=1.0, k_adiabatic=1.0)
    s = Solver(c, m)
    s.upload(u)
    t, _ = s.run(nsteps=2)
    ref, tr, _, _ = orc.Oracle.for_mesh(c, m).run(u, nsteps=2)
    assert t == tr and np.array_equal(s.download(), ref)


def test_repair_bit_exact():
    """Stages whose update leaves inadmissible nodes: in two layers of elements that the repair mends, and with a
    larger step in one that it cannot."""
    m = box()
    x = m.node_coords(setups.LGL4)[0]
    one = np.ones_like(x)
    u = np.ascontiguousarray(setups.prim2cons(one, 0 * one, 0 * one, 0 * one, np.where(x < 0.5, 10.0, 1.0), 1.4))
    c = abi.default_cfg(positivity=1)
    s = Solver(c, m)
    o = orc.Oracle.for_mesh(c, m)
    dt, _ = o.timestep(u)
    s.upload(u)
    uc, up = u.copy(), u.copy()
    assert s.stage(1, 96 * dt) == o.stage(uc, np.zeros_like(u), 0, 96 * dt) == 0
    orc.Oracle.for_mesh(abi.default_cfg(positivity=0), m).stage(up, np.zeros_like(u), 0, 96 * dt)
    assert not np.array_equal(uc, up)
    assert np.array_equal(s.download(), uc)
    s.upload(u)
    nbad = o.stage(u.copy(), np.zeros_like(u), 0, 128 * dt)
    with pytest.raises(abi.NemoError) as ei:
        s.stage(1, 128 * dt)
    assert ei.value.code == 4 and s.status()[1] == nbad > 0

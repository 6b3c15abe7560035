"""The plain FP64 stage kernel where its task layout and its own quotients could go wrong: meshes down to a
single element that is its own neighbour, odd element counts, domain boundaries, 2:1 faces, both kernels
(specialised and general) with and without blending; and states whose densities and pressures sit on and
next to 1 and 2, where a reciprocal rounds next to a tie.  Everything is compared with the FP64 oracle bit
for bit: the plain path's contract leaves no tolerance."""
import numpy as np
import pytest

from nemo_b200 import abi, mesh, setups
from nemo_b200.solver import Solver
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _fin():
    yield
    try:
        abi.call("nemo_gpu_finalize")
    except Exception:
        pass


MESHES = {
    "one periodic element": lambda: mesh.brick(1),
    "one open element": lambda: mesh.brick(1, periodic=(False,) * 3),
    "2x1x1": lambda: mesh.brick(2, 1, 1),
    "3x5x2, open in y": lambda: mesh.brick(3, 5, 2, periodic=(True, False, True)),
    "forest": lambda: mesh.forest(2, lambda lvl, c, s: c[:, 1] < 0.5, max_level=1),
}


@pytest.mark.parametrize("blend", [False, True])
@pytest.mark.parametrize("vf,sf", [(abi.VOLFLUX_CHANDRASHEKAR, abi.SURFFLUX_HLLC), (abi.VOLFLUX_CENTRAL, abi.SURFFLUX_RUSANOV)])
@pytest.mark.parametrize("name", list(MESHES))
def test_steps_bit_exact(name, vf, sf, blend):
    m = MESHES[name]()
    # a density jump between neighbouring nodes makes alpha > 0 in part of the elements
    u = setups.smooth_random(m, seed=5)
    u[:, :, 17] *= 1.5
    c = abi.default_cfg(volume_flux=vf, surface_flux=sf, indicator=abi.IND_MODAL if blend else abi.IND_NONE, positivity=1)
    s = Solver(c, m)
    o = orc.Oracle.for_mesh(c, m)
    s.upload(u)
    assert np.array_equal(s.rhs(), o.rhs(u, alpha=o.alpha(u)) if blend else o.rhs(u))
    t, n = s.run(nsteps=3)
    ref, tr, nr, _ = o.run(u, nsteps=3)
    assert t == tr and n == nr
    assert np.array_equal(s.download(), ref)


@pytest.mark.parametrize("sf", [abi.SURFFLUX_HLLC, abi.SURFFLUX_RUSANOV])
@pytest.mark.parametrize("base", [0.5, 1.0, 2.0])
def test_quotients_next_to_powers_of_two(base, sf):
    """Densities and pressures within a few ulp of a power of two, from below (significands of all ones) and
    from above, on nodes at rest and moving: every quotient of the fluxes meets its rounding ties."""
    m = mesh.brick(4)
    rng = np.random.default_rng(3)
    shape = (m.E, 64)

    def near(b):
        x = np.full(shape, b)
        k = rng.integers(-4, 5, size=shape)
        for _ in range(4):
            x = np.where(k > 0, np.nextafter(x, 9.0), np.where(k < 0, np.nextafter(x, 0.0), x))
            k = k - np.sign(k)
        return x

    v = [np.where(rng.random(shape) < 0.5, 0.0, rng.choice([0.25, 1.0, 2.0 ** -30, -0.5], size=shape)) for _ in range(3)]
    rho, p = near(base), near(base)
    rho[: m.E // 2] = near(1.0)[: m.E // 2]
    u = np.ascontiguousarray(setups.prim2cons(rho, v[0], v[1], v[2], p, 1.4))
    c = abi.default_cfg(surface_flux=sf, indicator=abi.IND_MODAL)
    s = Solver(c, m)
    s.upload(u)
    o = orc.Oracle.for_mesh(c, m)
    assert np.array_equal(s.rhs(), o.rhs(u, alpha=o.alpha(u)))


def mhd_state(m, seed, mu0):
    """Smooth periodic GLM-MHD state, every variable its own sinusoid, jumps between some nodes."""
    u5 = setups.smooth_random(m, seed=seed, kappa=5.0 / 3.0)
    x, y, z = m.node_coords(setups.LGL4)
    b = [0.3 + 0.2 * np.sin(2 * np.pi * (x + y)), -0.1 * np.cos(2 * np.pi * z), 0.15 * np.sin(2 * np.pi * (y - z))]
    psi = 0.02 * np.cos(2 * np.pi * x)
    b[0][:, 17] += 0.4
    u = np.concatenate([u5, np.stack(b + [psi])])
    u[4] += 0.5 / mu0 * (b[0] ** 2 + b[1] ** 2 + b[2] ** 2 + psi ** 2)
    u[:5, :, 17] *= 1.5
    u[4, :, 17] += 1.0
    return np.ascontiguousarray(u)


@pytest.mark.parametrize("blend", [False, True])
@pytest.mark.parametrize("vf,sf,mu0", [(abi.VOLFLUX_EC_MHD, abi.SURFFLUX_HLLD, 1.0), (abi.VOLFLUX_CENTRAL, abi.SURFFLUX_HLLD, 1.0),
                                       (abi.VOLFLUX_EC_MHD, abi.SURFFLUX_RUSANOV, 1.3)])
@pytest.mark.parametrize("name", list(MESHES))
def test_mhd_steps_bit_exact(name, vf, sf, mu0, blend):
    m = MESHES[name]()
    u = mhd_state(m, 5, mu0)
    c = abi.default_cfg(eqn=abi.EQN_MHD, n_vars=9, volume_flux=vf, surface_flux=sf, kappa=5.0 / 3.0, mu0=mu0, positivity=1,
                        indicator=abi.IND_MODAL if blend else abi.IND_NONE, glm_ch=0.7, glm_alpha=0.3)
    s = Solver(c, m)
    o = orc.Oracle.for_mesh(c, m)
    s.upload(u)
    assert np.array_equal(s.rhs(), o.rhs(u, alpha=o.alpha(u)) if blend else o.rhs(u))
    t, n = s.run(nsteps=3)
    ref, tr, nr, _ = o.run(u, nsteps=3)
    assert t == tr and n == nr
    assert np.array_equal(s.download(), ref)


@pytest.mark.parametrize("box", [(1, 1, 1), (3, 21, 1), (4, 4, 4), (5, 13, 1), (11, 31, 3), (16, 8, 8), (5, 5, 41), (3, 683, 1)])
def test_totals_at_chunk_edges(box):
    """Conserved totals around the element blocks (64) and the summation chunks (1024): 1, 63, 64, 65, 1023, 1024,
    1025 and 2049 elements, in the oracle's serial order bit for bit, Euler and GLM-MHD."""
    m = mesh.brick(*box)
    for mhd in (False, True):
        u = mhd_state(m, 2, 1.0) if mhd else setups.smooth_random(m, seed=2)
        c = abi.default_cfg(eqn=abi.EQN_MHD, n_vars=9, volume_flux=abi.VOLFLUX_EC_MHD, surface_flux=abi.SURFFLUX_HLLD) if mhd \
            else abi.default_cfg()
        s = Solver(c, m)
        s.upload(u)
        assert np.array_equal(s.totals(), orc.Oracle.for_mesh(c, m).totals(u)[: u.shape[0]])
        s.finalize()


@pytest.mark.parametrize("over", [0, 1])
@pytest.mark.parametrize("form", ["special", "general", "learned"])
def test_either_side_of_the_wide_kernels_limit(over, form):
    """The largest mesh that takes three directions at a time (12 elements per SM) and one element more, with every
    kind of kernel: specialised, general, learned indicator, and the rhs kernel."""
    import torch
    from nemo_b200 import learned
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    m = mesh.brick(12 * sms + over, 1, 1)
    u = setups.smooth_random(m, seed=3)
    u[:, :, 17] *= 1.5
    kw = dict(indicator=abi.IND_LEARNED if form == "learned" else abi.IND_MODAL, positivity=1)
    if form == "general":
        kw.update(surface_flux=abi.SURFFLUX_RUSANOV, volume_flux=abi.VOLFLUX_CENTRAL)
    c = abi.default_cfg(**kw)
    s = Solver(c, m)
    if form == "learned":
        learned.install()
        w, lo, hi, _ = learned.load()
        orc.set_mlp(learned.bf16_round(w), lo, hi)
    o = orc.Oracle.for_mesh(c, m)
    s.upload(u)
    assert np.array_equal(s.rhs(), o.rhs(u, alpha=o.alpha(u)))
    t, _ = s.run(nsteps=2)
    ref, tr, _, _ = o.run(u, nsteps=2)
    assert t == tr and np.array_equal(s.download(), ref)

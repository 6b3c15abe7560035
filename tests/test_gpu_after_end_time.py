"""Calls that follow a run which reached its end time: the device then holds its `done` mark, under which
stage kernels do nothing, but a launch that only prepares (indicator and CFL bound of the state) has to work
all the same.  Each call gives what it gives for the same state freshly uploaded, bit for bit; the plain
FP64 Euler form is also compared with the oracle."""
import numpy as np
import pytest

from nemo_b200 import abi, learned, mesh, setups
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


def case(mhd, precision):
    m = mesh.brick(4, lo=(-0.5,) * 3, hi=(0.5,) * 3)
    if mhd:
        c = abi.default_cfg(eqn=abi.EQN_MHD, n_vars=9, volume_flux=abi.VOLFLUX_EC_MHD, surface_flux=abi.SURFFLUX_HLLD,
                            kappa=5.0 / 3.0, indicator=abi.IND_MODAL, positivity=1, precision=precision)
        return c, m, setups.orszag_tang(m)
    c = abi.default_cfg(positivity=1, precision=precision, indicator=abi.IND_MODAL)
    return c, m, setups.sedov(m, sigma=0.1)


def at_end(c, m, u, t_end=1e-3):
    s = Solver(c, m)
    s.upload(u)
    t, n = s.run(t_end=t_end)
    assert t == t_end and n > 0
    return s


@pytest.mark.parametrize("precision", [abi.PREC_FP64, abi.PREC_FP32])
@pytest.mark.parametrize("mhd", [False, True])
def test_time_step_and_second_runs(mhd, precision):
    c, m, u = case(mhd, precision)
    s = at_end(c, m, u)
    u1 = s.download()
    bound = s.calc_timestep()
    s.run_async(2)
    s.sync()
    u2 = s.download()
    s = at_end(c, m, u)
    s.run_async(2)
    s.sync()
    assert np.array_equal(s.download(), u2)
    s = at_end(c, m, u)
    s.run(nsteps=2)
    assert np.array_equal(s.download(), u2)
    s.finalize()
    s = Solver(c, m)
    s.upload(u1)
    assert s.calc_timestep() == bound
    s.run(nsteps=2)
    assert np.array_equal(s.download(), u2)
    if not mhd and precision == abi.PREC_FP64:
        o = orc.Oracle.for_mesh(c, m)
        assert bound == o.timestep(u1)
        assert np.array_equal(o.run(u1, nsteps=2)[0], u2)


@pytest.mark.parametrize("precision", [abi.PREC_FP64, abi.PREC_FP32])
def test_new_weights(precision):
    """Weights installed after the end time: the coefficients and the rhs are the new indicator's."""
    m = mesh.brick(8)
    c = abi.default_cfg(positivity=1, precision=precision, indicator=abi.IND_LEARNED)   # modal until there are weights
    s = at_end(c, m, learned.random_problem(m, np.random.default_rng(1)))   # the indicators differ by up to 0.2 on it
    u1 = s.download()
    modal = s.alpha()
    learned.install()
    alpha, rhs = s.alpha(), s.rhs()
    assert not np.array_equal(alpha, modal)
    s.upload(u1)
    assert np.array_equal(alpha, s.alpha()) and np.array_equal(rhs, s.rhs())
    if precision == abi.PREC_FP64:
        w, lo, hi, _ = learned.load()
        orc.set_mlp(learned.bf16_round(w), lo, hi)
        o = orc.Oracle.for_mesh(c, m)
        a = o.alpha(u1)
        assert np.array_equal(alpha, a) and np.array_equal(rhs, o.rhs(u1, alpha=a))

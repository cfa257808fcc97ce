"""Red-black SOR solves where the sweeps on the change of p could part from the
scheme on p itself (k_sor_pass, the oracle): relaxation factors, scales of the
data and of the box, solves one after another, very unlike spacings."""
import numpy as np
import pytest

from conftest import rel_err

pytestmark = pytest.mark.gpu


def _sim(dims, length=(1.0, 1.0, 1.0), **keys):
    from nusif import Simulation
    from nusif.params import cavity
    return Simulation(cavity(dims, xlength=length[0], ylength=length[1], zlength=length[2], te=1e9,
                             **keys))


@pytest.mark.parametrize("arith", ["df32", "fp64"])
@pytest.mark.parametrize("dims", [(12, 12, 12), (40, 41, 39)])
def test_no_relaxation_runs_to_itermax(nusif_lib, oracle_mod, dims, arith):
    """omg 0: p stays, the residual too, and no iteration converges."""
    o = oracle_mod
    rng = np.random.default_rng(11)
    with _sim(dims, omg=0.0, eps=1e-6, itermax=7, arith=arith) as sim:
        p = rng.standard_normal(sim.padded_shape)
        rhs = rng.standard_normal(sim.padded_shape)
        sim.set_field("p", p)
        sim.set_field("rhs", rhs)
        res = sim.solve()
        it, want = o.op_solve_rb(o.grid(*dims), 1e-6, 0.0, 7, p, rhs)
        assert sim.iterations == it == 7
        assert res == pytest.approx(want, rel=1e-11)
        assert rel_err(sim.field("p"), p) < 1e-11

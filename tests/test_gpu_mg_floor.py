"""Where FP64 multigrid comes to rest: the true residual (long double) of the p it
leaves after more cycles than it needs, p large against its variation.

In units of diag ulp(|p|) / sqrt(12), the deviation of a rounding: a sweep
rounds a value when it stores it, its partial sums (a third, two thirds) and the
three neighbour sums (a third each), sqrt(17 / 9) together, times sqrt(7 / 6) by
the operator, 1.5; of a constant the partial sums round alike in all cells of a
colour, up to a quarter of a unit in the last place apart, which is 0.9 more:
2.5. Weights that do not add up to 1 leave more."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _true_residual(p, rhs, h):
    q = np.pad(p.astype(np.longdouble), 1, mode="edge")
    c = slice(1, -1)
    r = (rhs - rhs.mean()).astype(np.longdouble)
    for d, axis in zip(h, (2, 1, 0)):
        lo, hi = [c, c, c], [c, c, c]
        lo[axis], hi[axis] = slice(0, -2), slice(2, None)
        r -= (q[tuple(lo)] + q[tuple(hi)] - 2 * q[c, c, c]) / (np.longdouble(d) * np.longdouble(d))
    return float(np.sqrt((r * r).mean()))


@pytest.mark.parametrize("omega", [1.0, 1.3])
@pytest.mark.parametrize("dims", [(64, 64, 64), (96, 96, 96), (60, 44, 52), (48, 24, 72), (80, 16, 32)])
def test_true_residual_at_rest(nusif_lib, dims, omega):
    from nusif import Simulation
    from nusif.params import cavity
    rng = np.random.default_rng(1)
    offset = 1.03e6
    with Simulation(cavity(dims, te=1e9, solver="mg", mg_pre=2, mg_post=2, mg_omega=omega, rtol=1e-14,
                           mg_cycles=150)) as sim:
        c = (slice(1, -1),) * 3
        rhs = 100.0 * rng.standard_normal(sim.padded_shape)
        rhs -= rhs[c].mean()
        sim.set_field("p", np.full(sim.padded_shape, offset))
        sim.set_field("rhs", rhs)
        sim.solve()
        p = sim.field("p")[c]
        h = (sim.d.grid.dx, sim.d.grid.dy, sim.d.grid.dz)
    assert abs(p - offset).max() < 0.01 * offset
    unit = sum(2.0 / d ** 2 for d in h) * np.spacing(offset) / 12.0 ** 0.5
    assert _true_residual(p, rhs[c], h) < 2.5 * unit

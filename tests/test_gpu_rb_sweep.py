"""Red-black SOR by whole-iteration sweeps on the change of p, at the sizes
where its tiles can go wrong: one cell, rows of odd length (a pair without a
second column), rows cut into tiles (more than 128 cells), rows and planes
that end inside a block, and stops after the iterations that run on p itself.

Small grids run all iterations in one cluster of blocks: one block, several,
sixteen, the last slabs empty or not full, and the largest it takes.

Tolerance: an update rounds its operands to pairs, a few 2^-47 (7e-15) of the
largest pressure, and the iteration does not amplify it; 60 iterations of a
dozen such roundings stay below 60 * 12 * 7e-15 = 5e-12, so 1e-11.
"""
import numpy as np
import pytest

from conftest import rel_err

pytestmark = pytest.mark.gpu

DIMS = [(1, 1, 1), (1, 7, 4), (7, 1, 1), (3, 2, 40), (129, 5, 6), (131, 20, 9), (260, 33, 3),
        (64, 64, 64), (40, 41, 39), (5, 90, 33), (200, 160, 21)]


@pytest.mark.parametrize("arith", ["df32", "fp64"])
@pytest.mark.parametrize("dims", DIMS)
def test_sweeps_match_oracle(nusif_lib, oracle_mod, dims, arith):
    from nusif import Simulation
    from nusif.params import cavity
    o = oracle_mod
    rng = np.random.default_rng(3)
    for cube in (False, True):  # three spacings, or one
        length = [0.1 * n for n in dims] if cube else [1.0, 0.7, 1.3]
        vals = cavity(dims, xlength=length[0], ylength=length[1], zlength=length[2], omg=1.7,
                      eps=1e-9, itermax=60, arith=arith)
        with Simulation(vals) as sim:
            g = o.grid(*dims, *length)
            # each solve starts anew, ghosts unlike the cells beside them; the second
            # one knows the first one's count
            for itermax in (60, 59, 3, 2, 2, 1):
                sim.s.itermax = itermax
                p = rng.standard_normal(sim.padded_shape)
                rhs = rng.standard_normal(sim.padded_shape)
                sim.set_field("p", p)
                sim.set_field("rhs", rhs)
                res = sim.solve()
                it, res_c = o.op_solve_rb(g, vals["eps"], vals["omg"], itermax, p, rhs)
                assert sim.iterations == it
                assert res == pytest.approx(res_c, rel=1e-11)
                assert rel_err(sim.field("p"), p) < 1e-11


@pytest.mark.parametrize("arith", ["df32", "fp64"])
@pytest.mark.parametrize("dims", [(8, 8, 8), (12, 12, 12), (17, 16, 5), (20, 20, 20), (9, 73, 28),
                                  (64, 10, 61), (131, 21, 12), (33, 31, 30), (36, 36, 36)])
def test_cluster_matches_oracle(nusif_lib, oracle_mod, dims, arith):
    test_sweeps_match_oracle(nusif_lib, oracle_mod, dims, arith)

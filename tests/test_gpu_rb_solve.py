"""Red-black SOR solves where the sweeps on the change of p could part from the
scheme on p itself (k_sor_pass, the oracle): relaxation factors, scales of the
data and of the box, solves one after another, very unlike spacings."""
import ctypes as C
import subprocess
from pathlib import Path

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


# the update is linear: with rhs and eps times c and p times c a^2, a the edge of
# the box, the iterations and p / (c a^2) are the same
SCALES = [(a, c, e) for a in ("df32", "fp64")
          for c, e in [(1.0, 1.0), (1.0, 1e-5), (1.0, 1e-6), (1.0, 1e-7), (1.0, 1e-9), (1.0, 1e4),
                       (1e-14, 1.0), (1e3, 1e-6)]]
# (pressures below 2^-74 lose the low part of their pairs in the iteration on p itself)
SCALES += [("fp64", 1e-10, 1e-9), ("fp64", 1e-100, 1.0)]


def _scaled_solve(sim_keys, o, dims, data, box, eps, itermax, rough):
    rng = np.random.default_rng(5)
    shape = tuple(n + 2 for n in dims[::-1])
    p = data * box ** 2 * rough * rng.standard_normal(shape)
    rhs = data * rng.standard_normal(shape)
    rhs -= rhs[1:-1, 1:-1, 1:-1].mean()
    with _sim(dims, [box] * 3, omg=1.7, itermax=itermax, **sim_keys) as sim:
        sim.s.eps = eps
        sim.set_field("p", p)
        sim.set_field("rhs", rhs)
        res = sim.solve()
        it, want = o.op_solve_rb(o.grid(*dims, box, box, box), eps, 1.7, itermax, p, rhs)
        assert sim.iterations == it
        assert res == pytest.approx(want, rel=1e-9)
        assert rel_err(sim.field("p"), p) < 1e-11
        return it


@pytest.mark.parametrize("arith,data,box", SCALES)
@pytest.mark.parametrize("dims", [(24, 24, 24), (40, 41, 39)])
def test_iterations_do_not_depend_on_scale(nusif_lib, oracle_mod, dims, arith, data, box):
    """Boxes of micrometres in SI units, small and large data: the same count and
    residual as the oracle's, and p to the rounding of the unscaled solve."""
    it = _scaled_solve({"arith": arith}, oracle_mod, dims, data, box, 1e-4 * data, 600, 1e-3)
    assert 60 < it < 600


# squares whose sum over the grid, or (fp64) whose size, is beyond a float; nothing converges
@pytest.mark.parametrize("arith,data", [("df32", 1e17), ("fp64", 1e30)])
@pytest.mark.parametrize("dims", [(24, 24, 24), (40, 41, 39), (128, 96, 80)])
def test_large_residuals_run_on(nusif_lib, oracle_mod, dims, arith, data):
    assert _scaled_solve({"arith": arith}, oracle_mod, dims, data, 1.0, 0.25, 20, 1e-6) == 20


@pytest.fixture(scope="module")
def rb_exact(tmp_path_factory):
    """rb_exact.c as a function of (dims, length, omega, iterations, p, rhs), in place."""
    lib = tmp_path_factory.mktemp("rb") / "librb_exact.so"
    subprocess.run(["gcc", "-O2", "-fopenmp", "-shared", "-fPIC", str(Path(__file__).with_name("rb_exact.c")), "-o",
                    str(lib)], check=True)
    f = C.CDLL(str(lib)).rb_exact
    f.argtypes = [C.c_int] * 3 + [C.c_double] * 4 + [C.c_int] + [C.c_void_p] * 2

    def run(dims, h, omega, iterations, p, rhs):
        assert f(*dims, *h, omega, iterations, p.ctypes.data, rhs.ctypes.data) == 0

    return run


def _modes(dims, rng, count=8):
    """A smooth field without flux through the walls, padded, zero ghosts."""
    out = np.zeros([n + 2 for n in dims[::-1]])
    for _ in range(count):
        m = rng.integers(0, 5, 3)
        x, y, z = (np.cos(q * np.pi * (np.arange(n) + 0.5) / n) for q, n in zip(m, dims))
        out[1:-1, 1:-1, 1:-1] += (rng.standard_normal() / (1 + (m ** 2).sum()) *
                                  z[:, None, None] * y[None, :, None] * x[None, None, :])
    return out


def _error_against_64_bits(rb_exact, dims, length, iterations, p, rhs, omega=1.7, **keys):
    with _sim(dims, length, omg=omega, eps=1e-30, itermax=iterations, **keys) as sim:
        sim.set_field("p", p)
        sim.set_field("rhs", rhs)
        sim.solve()
        assert sim.iterations == iterations
        got = sim.field("p")
        g = sim.d.grid
        want = p.copy()
        rb_exact(dims, (g.dx, g.dy, g.dz), omega, iterations, want, rhs)
    c = (slice(1, -1),) * 3
    return rel_err(got[c], want[c])


# Tolerance: an iteration on p rounds p and its operands, to 2^-52 of the largest
# pressure (pairs: 2^-47), anew each time, and damps what the earlier ones left;
# independent errors add up to their size times the root of the count, twice
# that for the largest cell. (An error that is the same in every iteration adds
# up to the count.)
def _bound(iterations, arith):
    return 2.0 * iterations ** 0.5 * (2.0 ** -47 if arith == "df32" else 2.0 ** -52)


@pytest.mark.parametrize("arith", ["df32", "fp64"])
@pytest.mark.parametrize("dims,length", [((6, 160, 7), (4.0, 1.0, 1.0)),
                                         ((64, 64, 4), (0.01, 1.0, 1.0)),
                                         ((40, 12, 12), (30.0, 4.0, 4.0))])
def test_unlike_spacings_keep_their_factors(nusif_lib, rb_exact, dims, length, arith):
    """Spacings whose factors differ by orders of magnitude, from rest."""
    rng = np.random.default_rng(6)
    h2 = [(x / n) ** 2 for x, n in zip(length, dims)]
    rhs = _modes(dims, rng) / min(h2)
    err = _error_against_64_bits(rb_exact, dims, length, 500, np.zeros_like(rhs), rhs, arith=arith)
    assert err < _bound(500, arith)


def _laplacian(p, h2):
    """Of the interior of p, ghosts like the cells beside them; zero ghosts."""
    c = slice(1, -1)
    q = np.pad(p[c, c, c], 1, mode="edge")
    out = np.zeros_like(p)
    m = 2.0 * q[c, c, c]
    out[c, c, c] = ((q[c, c, :-2] + q[c, c, 2:] - m) / h2[0] +
                    (q[c, :-2, c] + q[c, 2:, c] - m) / h2[1] +
                    (q[:-2, c, c] + q[2:, c, c] - m) / h2[2])
    return out


@pytest.mark.parametrize("arith", ["df32", "fp64"])
@pytest.mark.parametrize("start", ["near", "far"])
@pytest.mark.parametrize("dims,length", [((24, 24, 24), (1.0, 1.0, 1.0)), ((6, 160, 7), (4.0, 1.0, 1.0)),
                                         ((42, 28, 30), (1.5, 1.5, 2.0)), ((40, 38, 36), (4.0, 3.8, 3.6)),
                                         ((131, 25, 16), (1.0, 1.0, 1.0))])
def test_change_of_p_keeps_the_bits_of_p(nusif_lib, rb_exact, dims, length, start, arith):
    """From a pressure near the end of the solve, where r0 is most of what
    there is, and from one that has nothing to do with it, where d is as large as p;
    by one cluster and by sweeps."""
    rng = np.random.default_rng(8)
    h2 = [(x / n) ** 2 for x, n in zip(length, dims)]
    p = _modes(dims, rng)
    rhs = rng.standard_normal(p.shape)
    if start == "near":
        rhs = _laplacian(p + 0.03 * _modes(dims, rng) + 1e-4 * rhs, h2)
    else:
        rhs -= rhs[1:-1, 1:-1, 1:-1].mean()
    n = 200
    assert _error_against_64_bits(rb_exact, dims, length, n, p, rhs, arith=arith) < _bound(n, arith)


# the last two: more block sums than a sweep's blocks fold by themselves
@pytest.mark.parametrize("arith", ["df32", "fp64"])
@pytest.mark.parametrize("dims", [(16, 16, 16), (40, 41, 39), (200, 40, 40), (2, 4000, 40),
                                  (1024, 1024, 1)])
def test_solves_do_not_depend_on_earlier_ones(nusif_lib, dims, arith):
    """The same p, rhs, eps and itermax give the same bits, whatever the solver
    ran before (its iteration count decides how many launches are queued)."""
    rng = np.random.default_rng(9)
    eps, itermax = 1e-9, 90
    with _sim(dims, [0.1 * n for n in dims], omg=1.7, eps=eps, itermax=itermax, arith=arith) as sim:
        p = rng.standard_normal(sim.padded_shape)
        rhs = rng.standard_normal(sim.padded_shape)

        def solve(eps, itermax):
            sim.s.eps, sim.s.itermax = eps, itermax
            sim.set_field("p", p)
            sim.set_field("rhs", rhs)
            return sim.solve(), sim.iterations, sim.field("p")

        first = solve(eps, itermax)  # a new solver's
        on_the_way = 4.0 * first[0] ** 0.5  # converges between two chunks' ends, or at one
        middle = solve(on_the_way, itermax)
        assert 2 < middle[1] < itermax
        for count in (2, 3, 1, 7, 16, middle[1], 40):
            solve(eps, count)
            for args, want in (((eps, itermax), first), ((on_the_way, itermax), middle)):
                got = solve(*args)
                assert got[:2] == want[:2]
                np.testing.assert_array_equal(got[2], want[2])


@pytest.mark.parametrize("arith", ["df32", "fp64"])
@pytest.mark.parametrize("dims", [(2, 4000, 40), (1024, 1024, 1), (1500, 900, 2)])
def test_long_lists_of_block_sums_match_oracle(nusif_lib, oracle_mod, dims, arith):
    """More than 1024 block sums: folded by a launch of its own."""
    from test_gpu_rb_sweep import test_sweeps_match_oracle
    test_sweeps_match_oracle(nusif_lib, oracle_mod, dims, arith)

"""The clusters of the coarse levels on grids that reach them: each test also
checks, by the names of the kernels that ran, that the cluster was one of them.
(Many grids end in a coarsest level of more than 1024 cells, which k_mg_bottom
does not take, or have one level only.)"""
import numpy as np
import pytest

from test_gpu_mg import _sim, test_mg_fp64_matches_oracle as mg_fp64_matches_oracle

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def profiler():
    """A profiler that has started: its first session can end without events."""
    import torch
    x = torch.zeros(1, device="cuda")
    for _ in range(10):
        with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
            x += 1.0
            torch.cuda.synchronize()
        if prof.key_averages():
            return
    pytest.fail("the profiler records no kernels")


def _solve(dims, solver, rtol, **keys):
    """(residual, cycles, p, names of the kernels) of a host-driven solve of random data."""
    import torch
    rng = np.random.default_rng(5)
    with _sim(dims, solver, rtol, mg_graph=0, **keys) as sim:
        sim.set_field("p", rng.standard_normal(sim.padded_shape))
        sim.set_field("rhs", rng.standard_normal(sim.padded_shape))
        with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
            res = sim.solve()
            torch.cuda.synchronize()
        names = {e.key for e in prof.key_averages()}
        return res, sim.iterations, sim.field("p"), names


def _ran(names, kernel):
    return any(kernel in n for n in names)


# rows of 24 and 12; x kept, y halved alone; y and z halved, then z alone, odd rows; an odd
# level below a halved one; all halved, then x alone; the largest inverse whose rows are
# copied to shared memory (640 cells), others are read where they are
@pytest.mark.parametrize("pre,post", [(1, 1), (2, 0), (3, 3), (1, 2)])
@pytest.mark.parametrize("dims", [(48, 16, 16), (12, 64, 8), (13, 16, 32), (26, 32, 32), (64, 32, 16),
                                  (40, 16, 16), (36, 36, 36)])
def test_bottom_cluster_matches_per_level_kernels(nusif_lib, dims, pre, post):
    """The same bits as a kernel per sweep and transfer (mg_tail 1: no level is that small)."""
    out = [_solve(dims, "mg-mixed", 1e-9, mg_pre=pre, mg_post=post, mg_omega=1.2, mg_cycles=3,
                  mg_tail=tail) for tail in (0, 1)]
    assert _ran(out[0][3], "k_mg_bottom") and not _ran(out[1][3], "k_mg_bottom")
    assert out[0][:2] == out[1][:2]
    np.testing.assert_array_equal(out[0][2], out[1][2])


# coarsest levels of 31 x 41 x 2 and 31 x 17 x 8 (slabs of one plane, blocks without cells),
# 9 x 10 x 12 (whole slabs of two), 33 x 31 x 15 (almost the 16384 cells that a cluster takes)
# and 33 x 31 x 17 (beyond: sweeps in global memory)
@pytest.mark.parametrize("dims,cluster", [((62, 82, 2), True), ((62, 34, 8), True), ((36, 20, 48), True),
                                          ((66, 62, 15), True), ((66, 62, 17), False)])
def test_coarsest_fp64_sweeps_match_oracle(nusif_lib, oracle_mod, dims, cluster):
    names = _solve(dims, "mg", 1e-6)[3]
    assert _ran(names, "k_mg_prolong")  # two levels at least
    assert _ran(names, "k_mg_coarse_f64") == cluster
    mg_fp64_matches_oracle(nusif_lib, oracle_mod, dims)

"""The step's reductions allocate nothing once a simulation exists: grids whose
reductions use different numbers of blocks, under stream capture, which forbids
allocation."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(8, 8, 8), (17, 16, 5), (32, 32, 32), (64, 48, 50), (96, 96, 96)])
def test_normalize_pressure_under_capture(nusif_lib, dims):
    import torch

    from nusif import Simulation
    from nusif.params import cavity
    rng = np.random.default_rng(3)
    with Simulation(cavity(dims, te=1e9)) as sim:
        p = rng.standard_normal(sim.padded_shape)
        sim.compute_timestep()  # a reduction of another size
        sim.set_field("p", p)
        graph = torch.cuda.CUDAGraph()
        try:
            with torch.cuda.graph(graph):
                nusif_lib.nusifSetStream(torch.cuda.current_stream().cuda_stream)
                sim.normalize_pressure()
        finally:
            nusif_lib.nusifSetStream(None)
        graph.replay()
        torch.cuda.synchronize()
        got = sim.field("p")
        sim.set_field("p", p)
        sim.normalize_pressure()
        np.testing.assert_array_equal(got, sim.field("p"))
        c = (slice(1, -1),) * 3
        assert abs(got[c].mean()) < 1e-13

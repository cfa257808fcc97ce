"""All six velocity boundary faces in one launch against the oracle, which
applies them in the reference's order: every pair of conditions on every pair
of faces, on grids whose axes are short enough that all edges and corners
matter (and with an axis of one cell, which takes one launch per face). Copies
and sign changes: exact, signs of zeros included."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SLOTS = ["bcLeft", "bcRight", "bcBottom", "bcTop", "bcFront", "bcBack"]


@pytest.mark.parametrize("dims", [(2, 2, 2), (3, 2, 4), (5, 33, 9), (1, 3, 2), (4, 1, 3), (3, 4, 1)])
def test_faces_match_oracle(nusif_lib, oracle_mod, dims):
    from nusif import Simulation
    from nusif.params import cavity
    rng = np.random.default_rng(5)
    combos = set()
    for a in range(6):
        for b in range(a):
            for ca in range(1, 5):
                for cb in range(1, 5):
                    bc = list(rng.integers(1, 5, 6))
                    bc[a], bc[b] = ca, cb
                    combos.add(tuple(int(c) for c in bc))
    with Simulation(cavity(dims, te=1e9)) as sim:
        g = oracle_mod.grid(*dims)
        fields = {f: rng.standard_normal(sim.padded_shape) for f in "uvw"}
        for bc in sorted(combos):
            for slot, c in zip(SLOTS, bc):
                setattr(sim.d, slot, c)
            want = {f: a.copy() for f, a in fields.items()}
            for f, a in fields.items():
                sim.set_field(f, a)
            sim.set_boundary_conditions()
            oracle_mod.op_set_bc(g, bc, *(want[f] for f in "uvw"))
            for f in "uvw":
                got = sim.field(f)
                np.testing.assert_array_equal(got.view(np.int64), want[f].view(np.int64), err_msg=str(bc))

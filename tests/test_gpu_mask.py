"""GPU test of the masks built on the device: a new volume's (fluid except the y = 0 floor) and a caller's
bytes, of which any but 0 is fluid."""
import numpy as np
import pytest

import smoke_simulation_gb300 as smk

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(1, 1, 1), (3, 2, 5), (64, 4, 3), (65, 5, 2), (130, 37, 9)])
def test_masks_equal_their_definition(gpu, dims):
    nx, ny, nz = dims
    sim = smk.Simulation(nx, ny, nz)
    want = np.ones((nz, ny, nx), np.uint8)
    want[:, 0, :] = 0
    assert np.array_equal(sim.read_state()["s"], want)
    mask = np.random.default_rng(3).choice(np.array([0, 1, 2, 128, 255], np.uint8), (nz, ny, nx))
    sim.set_mask(mask)
    assert np.array_equal(sim.read_state()["s"], (mask != 0).astype(np.uint8))
    sim.close()

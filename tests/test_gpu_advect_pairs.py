"""GPU test of the two advections' two-row forms (the density's strips of columns with a lone last row): tiles with and without positions at the clamp,
backtraces below, around and above the reach of its window within one warp, one-plane chunks up to
sixteen-plane ones, and velocities that are infinite or NaN, against the restatement of the step."""
import numpy as np
import pytest

import smoke_simulation_gb300 as smk
from oracle import oracle as O
from smoke_simulation_gb300 import scenes as S
from tests import helpers as H

pytestmark = pytest.mark.gpu


def _same(a, b):
    nan = np.isnan(b)  # a NaN's sign and payload are not the restatement's to fix
    return np.array_equal(np.isnan(a), nan) and np.array_equal(a[~nan].view(np.uint32), b[~nan].view(np.uint32))


@pytest.mark.parametrize("dims,reach,special", [
    ((6, 5, 7), 0.5, False),
    ((33, 18, 9), 1.5, False),      # one column and one row past a tile
    ((66, 35, 11), 0.3, False),     # exactly one tile without clamps
    ((67, 51, 40), 2.5, False),     # near and far backtraces in the same warps
    ((67, 51, 40), 0.89, True),
    ((131, 6, 12), 1.1, False),     # two full strips and one column more, an even number of rows
    ((24, 9, 21), 4.0, True),
    ((200, 120, 70), 1.2, True),    # longer chunks
])
def test_advection_equals_restatement(gpu, dims, reach, special):
    sc = S.small_scene(*dims, steps=2, seed=9, iterations=1, obstacles=1 if min(dims) > 8 else 0, noise=0.0)
    rng = np.random.default_rng(4)
    out = []
    for _ in range(3):
        a = (rng.uniform(-1.0, 1.0, sc.face_shape) * reach / sc.dt).astype(np.float32)
        if special:
            at = rng.integers(0, 4000, sc.face_shape)
            a[at == 0] = np.nan
            a[at == 1] = np.inf
            a[at == 2] = -np.inf
            a[at == 3] = 0.9 / sc.dt
        out.append(a)
    sc.u0, sc.v0, sc.w0 = out
    sim, o = smk.from_scene(sc), O.OracleSim(sc)
    for k in range(sc.steps):
        sim.step(sc.dt)
        o.step()
        a, b = sim.read_state(), H.oracle_state(o)
        for f in ("u", "v", "w", "rho"):
            for j in range(2):
                assert _same(np.asarray(a[f][j]), np.asarray(b[f][j])), (k, f, j)
    sim.close()

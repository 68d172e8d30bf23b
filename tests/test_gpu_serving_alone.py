"""GPU test of the streams form's switch between a lone request's solves (resident, the whole chip) and
shared ones: requests that start alone, are joined, and are left alone again give what the same grid
gives stepped by itself."""
import numpy as np
import pytest

import smoke_simulation_gb300 as smk
from smoke_simulation_gb300 import scenes as S, serving

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("steps,joined_at,joiner_steps", [(40, 6, 5), (12, 6, 20), (9, 0, 3)])
@pytest.mark.parametrize("storage", [smk.STORAGE_F32, smk.STORAGE_BF16_VEL])
def test_alone_joined_alone_equals_stepping(gpu, steps, joined_at, joiner_steps, storage):
    a = S.small_scene(44, 37, 41, seed=3, scheme=1, iterations=60, tol=1e-4, check_every=6, warm_start=1, steps=steps)
    b = S.small_scene(30, 52, 26, seed=4, scheme=1, iterations=60, tol=1e-4, check_every=6, warm_start=1,
                      steps=joiner_steps)
    for sc in (a, b):  # a request has no initial velocity
        sc.u0 = sc.v0 = sc.w0 = None
    srv = serving.Server()
    ids = [srv.submit(a, storage=storage)]
    for _ in range(joined_at):
        srv.tick()
    ids.append(srv.submit(b, storage=storage))
    srv.run_until_idle()
    for sc, rid in zip((a, b), ids):
        assert srv.status(rid)[0] == serving.REQ_DONE
        sim = smk.from_scene(sc, storage=storage)
        for _ in range(sc.steps):
            sim.step(sc.dt)
        assert np.array_equal(srv.outputs[rid].view(np.uint32), sim.read_density().view(np.uint32))
        sim.close()
    srv.close()

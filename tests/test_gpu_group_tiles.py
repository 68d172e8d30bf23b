"""GPU test of the grouped stages' tiles: more grids than one search step tells apart, members without
tiles in a stage (a grid of two cells on an axis), both output types of the velocity advection in one
batch, the blocked and the cooperative projection; every member equals the same grid stepped alone."""
import pytest

import smoke_simulation_gb300 as smk
from smoke_simulation_gb300 import scenes as S
from tests import helpers as H

pytestmark = pytest.mark.gpu

STORAGES = (smk.STORAGE_F32, smk.STORAGE_BF16, smk.STORAGE_BF16_VEL)


def _member(i):
    dims = (5 + (7 * i) % 31, 4 + (5 * i) % 23, 6 + (3 * i) % 19)
    if i % 13 == 4:
        return S.Scene("thin%d" % i, 2, 6, 9, dt=0.05, steps=1, scheme=1, iterations=12, tol=1e-4, check_every=4)
    if i == 9:
        dims = (140, 37, 30)
    return S.small_scene(*dims, seed=40 + i, scheme=1, iterations=12, tol=1e-4, check_every=4, obstacles=0, noise=0.6)


@pytest.mark.parametrize("count", [1, 33, 70])
@pytest.mark.parametrize("blocked", [0, 17, 137])  # the cap of the z-chunks: few grids get shorter ones
def test_grouped_tiles_equal_alone(gpu, count, blocked):
    scs = [_member(i) for i in range(count)]
    kinds = [STORAGES[(i // 2) % 3] for i in range(count)]
    a = [smk.from_scene(sc, report_div=1, storage=k) for sc, k in zip(scs, kinds)]
    b = [smk.from_scene(sc, report_div=1, storage=k) for sc, k in zip(scs, kinds)]
    batch = smk.Batch(a, mode=smk.BATCH_GROUPED)
    if blocked:
        batch.set_blocked(blocked)
        assert batch.blocked() == blocked
    else:
        batch.set_schedule(0, 4, 0)
    for _ in range(3):
        batch.step(0.05)
        for s in b:
            s.step(0.05)
    for i in range(count):
        assert H.first_mismatch(a[i].read_state(), b[i].read_state()) == "", i
        sa, sb = a[i].stats(), b[i].stats()
        assert (sa.sweeps, sa.div_max) == (sb.sweeps, sb.div_max), i
    batch.close()
    for s in a + b:
        s.close()

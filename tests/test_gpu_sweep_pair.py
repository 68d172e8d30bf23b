"""The blocked pressure sweep's pair form at the sizes where it can go wrong: every depth, chunks of
odd and even length, windows whose last tile holds one row or column, grids of odd sides, partial
launches and checks, against one colour pass per launch (which the other tests hold to the oracle)."""
import numpy as np
import pytest

import smoke_simulation_gb300 as smk
from smoke_simulation_gb300 import scenes as S
from tests import helpers as H


@pytest.mark.gpu
@pytest.mark.parametrize("dims", [(64, 48, 20), (65, 49, 21), (57, 41, 37), (113, 81, 19), (130, 45, 33), (17, 130, 9),
                                  (3, 3, 3), (9, 200, 5)])
@pytest.mark.parametrize("shape", [(4, 1), (4, 8), (4, 13), (4, 400), (6, 5), (6, 16), (2, 7), (2, 64)])
def test_pair_form_equals_one_pass_per_launch(gpu, dims, shape):
    # 14 sweeps: groups of 5 (10 passes: a partial launch first at depths 4 and 6), checked, then
    # a last group of 4; the second step's solve starts from the first one's pressure
    sc = S.small_scene(*dims, steps=3, seed=sum(dims), scheme=1, iterations=14, tol=1e-6, check_every=5, obstacles=1,
                       warm_start=1) if min(dims) > 4 else S.Scene("tiny", *dims, dt=0.05, steps=3, scheme=1,
                                                                   iterations=14, tol=1e-6, check_every=5, warm_start=1,
                                                                   spheres=[(1.0, 1.0, 1.0, 2.0)])
    sc.mask = S.bernoulli_mask(*dims, 0.05, seed=3)
    sc.obstacles = []
    a, b = (smk.from_scene(sc, report_div=1) for _ in range(2))
    a.set_sweep_kernel(*shape)
    b.set_sweep_kernel(0, 1)
    for k in range(sc.steps):
        a.step(sc.dt)
        b.step(sc.dt)
        sa, sb = a.stats(), b.stats()
        assert (sa.sweeps, sa.converged) == (sb.sweeps, sb.converged), k
        assert H.bits_equal(np.float32(sa.resid_max), np.float32(sb.resid_max)), k
        assert H.first_mismatch(a.read_state(), b.read_state()) == "", k
    a.close()
    b.close()


@pytest.mark.gpu
def test_values_that_are_not_finite_stay_where_they_were(gpu):
    """An infinity and a NaN in the field reach the same cells as with one pass per launch (a cell
    that is not projectable keeps its value whatever its neighbours hold)."""
    sc = S.small_scene(66, 50, 30, steps=1, seed=4, scheme=1, iterations=6, obstacles=0)
    sc.mask = S.bernoulli_mask(66, 50, 30, 0.1, seed=5)
    sc.u0[10, 12, 20] = np.inf
    sc.v0[15, 30, 40] = np.nan
    for shape in ((4, 8), (6, 30), (2, 11)):
        a, b = smk.from_scene(sc), smk.from_scene(sc)
        a.set_sweep_kernel(*shape)
        b.set_sweep_kernel(0, 1)
        a.step(sc.dt)
        b.step(sc.dt)
        x, y = a.read_state(), b.read_state()
        for f in ("rho", "u", "v", "w"):
            for p in range(2):
                assert np.array_equal(np.isnan(x[f][p]), np.isnan(y[f][p])), (shape, f)
                ok = ~np.isnan(y[f][p])
                assert np.array_equal(x[f][p][ok], y[f][p][ok]), (shape, f)
        a.close()
        b.close()

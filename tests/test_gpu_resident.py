"""Solves resident in shared memory (the form that small and middle grids take by themselves) against one
colour pass per launch, which the other tests hold to the oracle: the same bits on every field, sweep
counts and residuals included, at the sizes where boxes, sides and slots begin and end."""
import numpy as np
import pytest

import smoke_simulation_gb300 as smk
from smoke_simulation_gb300 import scenes as S
from tests import helpers as H
from tests.test_gpu_velocity_blocked import _special

DIMS = [(3, 3, 3), (4, 3, 5), (3, 40, 4), (5, 64, 3), (16, 17, 18), (33, 31, 29), (64, 64, 64), (65, 63, 66), (200, 9, 41),
        (80, 81, 79), (97, 61, 113), (100, 101, 99), (127, 126, 125), (128, 128, 128), (350, 40, 45)]


def _scene(dims, **kw):
    sc = S.Scene("resident", *dims, dt=0.05, steps=3, **kw)
    sc.mask = S.bernoulli_mask(*dims, 0.05, seed=sum(dims))
    sc.spheres = [(dims[0] // 2, dims[1] // 2, dims[2] // 2, 2.0)]
    sc.u0, sc.v0, sc.w0 = S.noise_velocity(sc.face_shape, 0.5, seed=7)
    return sc


@pytest.mark.gpu
@pytest.mark.parametrize("dims", DIMS)
@pytest.mark.parametrize("tol,storage", [(0.0, 0), (2e-2, 0), (1e-9, 2)])
def test_pressure_solve_equals_one_pass_per_launch(gpu, dims, tol, storage):
    sc = _scene(dims, scheme=1, iterations=13, tol=tol, check_every=4, warm_start=1, omega_warm=1.7,
                warm_extrapolate=0.5)
    a, b = (smk.from_scene(sc, storage=storage, report_div=1) for _ in range(2))
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
@pytest.mark.parametrize("dims", DIMS)
@pytest.mark.parametrize("iterations,omega,special", [(9, 1.9, False), (6, 1.9, True), (5, 1.37123456789, True)])
def test_velocity_passes_equal_one_pass_per_launch(gpu, dims, iterations, omega, special):
    sc = _scene(dims, iterations=iterations, omega=omega)
    if special:
        sc.u0, sc.v0, sc.w0 = _special(sc, 3)
    a, b = smk.from_scene(sc), smk.from_scene(sc)
    b.set_velocity_sweep(0)
    for k in range(2):
        a.step(sc.dt)
        b.step(sc.dt)
        assert H.first_mismatch(a.read_state(), b.read_state()) == "", k
    a.close()
    b.close()


@pytest.mark.gpu
def test_forms_may_change_between_steps_and_streams(gpu):
    """Resident steps, a set shape, a batch's branches and a restart of the pressure history in one
    simulation, on two streams, give what one pass per launch gives; autotuning keeps a form that
    does."""
    import torch
    sc = _scene((70, 50, 60), scheme=1, iterations=24, tol=1e-3, check_every=6, warm_start=1)
    a, b, c = (smk.from_scene(sc) for _ in range(3))
    b.set_sweep_kernel(0, 1)
    c.set_sweep_kernel(0, 1)
    pair = smk.Batch([a, c], mode=smk.BATCH_BRANCHES)
    streams = [torch.cuda.Stream() for _ in range(2)]
    for k, how in enumerate(["alone", "alone", "batch", "alone", "tuned", "alone", "write", "alone"]):
        st = streams[k % 2].cuda_stream
        torch.cuda.synchronize()
        if how == "tuned":
            a.autotune()
        if how == "write":
            state = b.read_state()
            a.write_state(state)
            b.write_state(state)
        if how == "batch":
            pair.step(sc.dt, st)
        else:
            a.step(sc.dt, st)
        b.step(sc.dt, st)
        torch.cuda.synchronize()
        assert H.first_mismatch(a.read_state(), b.read_state()) == "", (k, how)
        assert a.stats().sweeps == b.stats().sweeps, (k, how)
    pair.close()
    for s in (a, b, c):
        s.close()


@pytest.mark.gpu
@pytest.mark.parametrize("graphs", [True, False])
def test_resident_solves_on_several_streams_at_once(gpu, graphs):
    """Simulations stepped on their own streams, their resident solves (each a cooperative launch over the
    whole chip) in flight together: the same fields as stepped one after another."""
    import torch
    scs = [S.small_scene(60 + 9 * i, 52, 47 + 5 * i, seed=30 + i, iterations=12, obstacles=1, scheme=i % 2, tol=0.0)
           for i in range(4)]
    a, b = [smk.from_scene(sc) for sc in scs], [smk.from_scene(sc) for sc in scs]
    streams = [torch.cuda.Stream() for _ in scs]
    for s in a:
        s.set_graphs(graphs)
    for _ in range(12):
        for s, sc, st in zip(a, scs, streams):
            s.step(sc.dt, st.cuda_stream)
    torch.cuda.synchronize()
    for s, sc in zip(b, scs):
        for _ in range(12):
            s.step(sc.dt)
    for i, (x, y) in enumerate(zip(a, b)):
        x.sync()
        assert H.first_mismatch(x.read_state(), y.read_state()) == "", i

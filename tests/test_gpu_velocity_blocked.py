"""The velocity sweep that a REFERENCE-scheme simulation picks from its grid (temporally blocked on
large grids) against one colour pass per launch, which the other tests hold to the oracle: the same
bits on every field, with values on which its arithmetic takes its other paths."""
import ctypes as C

import numpy as np
import pytest

import smoke_simulation_gb300 as smk
from smoke_simulation_gb300 import scenes as S
from tests import helpers as H


def _special(sc, seed):
    """Velocities with zeros of both signs, subnormals, tiny and ordinary values."""
    rng = np.random.default_rng(seed)
    out = []
    for _ in range(3):
        a = rng.uniform(-1.0, 1.0, sc.face_shape).astype(np.float32)
        kind = rng.integers(0, 8, sc.face_shape)
        a[kind == 0] = 0.0
        a[kind == 1] = -0.0
        a[kind == 2] *= np.float32(2.0**-110)
        a[kind == 3] *= np.float32(2.0**-130)
        a[kind == 4] = (rng.integers(-40, 40, sc.face_shape)[kind == 4] * 1e-45).astype(np.float32)
        out.append(a)
    # a region that holds nothing else than such values
    for a in out:
        a[: sc.nz // 2][np.abs(a[: sc.nz // 2]) > 1e-20] = 0.0
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("dims,iterations,omega,special,depth", [
    ((130, 118, 141), 30, 1.9, False, 4),   # 60 passes: fourteen launches of 4 and two of 2
    ((130, 118, 141), 7, 1.9, True, 4),     # 14 passes: 4, 4, 4, 2
    ((257, 97, 115), 6, 1.9, True, 4),      # windows along x that end one column past a tile
    ((143, 145, 121), 5, 1.37123456789, False, 4),  # an over-relaxation without a small denominator
    ((113, 145, 121), 5, 1.37123456789, False, 0),  # resident in shared memory
])
def test_grid_choice_equals_one_pass_per_launch(gpu, dims, iterations, omega, special, depth):
    sc = S.small_scene(*dims, steps=2, seed=5, iterations=iterations, obstacles=2, omega=omega)
    if special:
        sc.u0, sc.v0, sc.w0 = _special(sc, 8)
    a, b = smk.from_scene(sc), smk.from_scene(sc)
    b.set_velocity_sweep(0)
    assert a.velocity_sweep()[0] == depth and b.velocity_sweep()[0] == 0
    for k in range(sc.steps):
        a.step(sc.dt)
        b.step(sc.dt)
        msg = H.first_mismatch(a.read_state(), b.read_state())
        assert msg == "", "step %d: %s" % (k, msg)
    # a switch to the warm-started pressure form goes on as after one pass per launch
    for s in (a, b):
        s.set_params(projection=smk.PROJECT_PRESSURE, warm_start=1, max_sweeps=8, omega=1.9, omega_warm=1.7,
                     omega_warm_after=3, warm_extrapolate=0.5)
    for k in range(3):
        a.step(sc.dt)
        b.step(sc.dt)
        assert H.first_mismatch(a.read_state(), b.read_state()) == "", k
    # and the pressure history then stays: the sweep no longer uses the pressure buffers
    for s in (a, b):
        s.set_params(projection=smk.PROJECT_REFERENCE)
    assert a.velocity_sweep()[0] == 0
    a.close()
    b.close()


@pytest.mark.parametrize("omega", [1.9, 1.85, 1.725, 1.9000001, 1.37123456789, 1.5 + 2.0**-50, -1.9, 2.0**-30])
def test_cell_arithmetic_for_any_omega(smoke_lib, omega):
    """float(double(x / d) * omega) for omegas with and without a small denominator."""
    fn = smoke_lib.smk_test_exact_cell
    fn.restype = C.c_int
    fn.argtypes = [C.c_void_p, C.c_void_p, C.c_int, C.c_double, C.c_void_p]
    rng = np.random.default_rng(3)
    x = rng.integers(0, 2**32, 1 << 17, dtype=np.uint64).astype(np.uint32)
    near = (rng.integers(0, 1 << 23, 1 << 17) + (127 << 23)).astype(np.uint32)  # ordinary significands
    small = rng.integers(1, 32 << 23, 1 << 16).astype(np.uint32)                # tiny and subnormal
    x = np.concatenate([x, near, small]).view(np.float32)
    x = np.ascontiguousarray(x[~np.isnan(x)])
    for d in range(1, 7):
        dd = np.full(x.size, d, np.int32)
        out = np.empty_like(x)
        assert fn(x.ctypes.data, dd.ctypes.data, x.size, omega, out.ctypes.data) == 0
        with np.errstate(over="ignore", invalid="ignore"):
            want = ((x / np.float32(d)).astype(np.float64) * omega).astype(np.float32)
        bad = np.flatnonzero(out.view(np.uint32) != want.view(np.uint32))
        assert bad.size == 0, (omega, d, x[bad[:4]], out[bad[:4]], want[bad[:4]])

"""The FP64 divergence measurement of the refinement: the maximum it reports is that of numpy's
float64 sums over the projected velocities, bit for bit as float, on rows that end anywhere in a
group of four cells."""
import numpy as np
import pytest

import smoke_simulation_gb300 as smk
from smoke_simulation_gb300 import scenes as S


@pytest.mark.gpu
@pytest.mark.parametrize("dims", [(3, 3, 3), (5, 4, 6), (13, 9, 7), (64, 5, 5), (131, 20, 18), (200, 70, 66)])
@pytest.mark.parametrize("noise", [0.5, 1e6, 1e-30, 3e-39])  # the last two: partial sums near and below 2^-126
def test_measured_divergence_is_numpys_float64(gpu, dims, noise):
    sc = S.Scene("m", *dims, dt=0.05, steps=1, scheme=1, iterations=6, tol=1e-12, check_every=3, refine=1,
                 refine_sweeps=2, clamp_mode=2)
    sc.mask = S.bernoulli_mask(*dims, 0.1, seed=1)
    sc.u0, sc.v0, sc.w0 = S.noise_velocity(sc.face_shape, noise, seed=2)
    sim = smk.from_scene(sc)
    sim.step(sc.dt)
    st = sim.read_state()
    u, v, w = (st[k][st["index_now"]].astype(np.float64) for k in "uvw")
    nx, ny, nz = dims
    c = (slice(0, nz), slice(0, ny), slice(0, nx))
    d = ((((-u[c] + u[:nz, :ny, 1:]) + -v[c]) + v[:nz, 1:, :nx]) + -w[c]) + w[1:, :ny, :nx]
    s = np.pad(st["s"] != 0, 1)
    nbrs = sum(s[1 + a:1 + a + nz, 1 + b:1 + b + ny, 1 + e:1 + e + nx].astype(int)
               for a, b, e in ((0, 0, 1), (0, 0, -1), (0, 1, 0), (0, -1, 0), (1, 0, 0), (-1, 0, 0)))
    live = (st["s"] != 0) & (nbrs > 0)
    inner = np.zeros_like(live)
    inner[1:-1, 1:-1, 1:-1] = True
    live &= inner
    want = np.float32(np.abs(d[live]).max()) if live.any() else np.float32(0)
    assert np.float32(sim.stats().div64_max).view(np.uint32) == want.view(np.uint32)
    sim.close()

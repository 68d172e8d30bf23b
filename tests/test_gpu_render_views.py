"""GPU tests of the renderer's ray-to-plane range, its per-block plane table, its remainder-step
quotients and its short cut through empty space: views for which the
range could cut a plane that the ray meets (an eye inside the box or far away, rays along the planes or
along the box sides, a box off the origin, a single plane, more planes than the table holds) equal the
CPU restatement, which tests every plane of every ray with plain divisions; so do lengths beyond the
quotients' range, and densities that are empty in part, negative, above one or infinite."""
import numpy as np
import pytest

import smoke_simulation_gb300 as smk
from oracle import oracle as O

pytestmark = pytest.mark.gpu

VIEWS = {
    "eye_in_box": dict(camera_pos=(3.0, -2.0, 5.0), camera_dir=(0.2, 0.1, -1.0)),
    "light_in_box": dict(light_pos=(4.0, 6.0, -3.0)),
    "far_eye": dict(camera_pos=(0.0, 300.0, 2900.0), camera_dir=(0.0, -0.1, -1.0), fovy_deg=1.5, zfar=5000.0),
    "along_axis": dict(camera_pos=(0.0, 0.0, 90.0), camera_dir=(0.0, 0.0, -1.0), light_pos=(0.0, 0.0, 80.0)),
    "half_vector_across": dict(camera_pos=(0.0, 0.0, 90.0), camera_dir=(0.0, 0.0, -1.0), light_pos=(90.0, 0.0, 0.0)),
    "box_off_origin": dict(box_pos=(7.0, -11.0, 4.0), camera_pos=(60.0, 40.0, 70.0), camera_dir=(-60.0, -45.0, -70.0)),
    "looks_away": dict(camera_dir=(1.0, 0.2, 0.1)),
    "one_plane": dict(planes=1),
    "past_the_table": dict(planes=2100, light_res=16, width=40, height=24),
    "tiny_near": dict(znear=1e-9, light_znear=1e-9),
    "far_lengths": dict(cell_size=1e8, camera_pos=(1e8, 2e9, 1e10), camera_dir=(0.0, -0.2, -1.0), light_pos=(1.2e10, 8e9, 0.0),
                        zfar=1e13, light_zfar=1e13),
    "wide": dict(fovy_deg=150.0, light_fovy_deg=120.0),
}


@pytest.mark.parametrize("view", sorted(VIEWS))
@pytest.mark.parametrize("n", [(33, 40, 27)])
def test_render_views_bit_exact_with_restatement(gpu, view, n):
    nx, ny, nz = n
    z, y, x = np.mgrid[0:nz, 0:ny, 0:nx]
    rho = (0.05 + 0.5 * np.sin(0.9 * x) ** 2 * np.cos(0.7 * y) ** 2 * np.sin(0.5 + 0.4 * z) ** 2).astype(np.float32)
    _same_as_restatement(rho, VIEWS[view])


@pytest.mark.parametrize("light", [(120.0, 80.0, 0.0), (0.0, 20.0, -120.0)])  # front-to-back, back-to-front
@pytest.mark.parametrize("density", ["islands", "negative", "negative_zero", "above_one", "infinite"])
def test_render_empty_space_bit_exact_with_restatement(gpu, density, light):
    z, y, x = np.mgrid[0:24, 0:31, 0:29]
    rho = np.where((x // 5 + y // 7 + z // 6) % 3 == 0, 0.4 + 0.02 * x, 0.0).astype(np.float32)
    if density == "negative":
        rho[(x + y + z) % 4 == 0] = -0.3
    elif density == "negative_zero":
        rho[rho == 0.0] = -0.0
        rho[:, 12:, :] = 0.0
    elif density == "above_one":
        rho *= 4.0
    elif density == "infinite":
        rho[9, 14, 11] = np.inf
    _same_as_restatement(rho, dict(light_pos=light))


def _same_as_restatement(rho, view):
    nz, ny, nx = rho.shape
    sim = smk.Simulation(nx, ny, nz)
    sim.set_density(rho)
    rp = smk.default_render_params(width=96, height=64, light_res=48, planes=37)
    for k, v in view.items():
        if isinstance(v, tuple):
            getattr(rp, k)[:] = v
        else:
            setattr(rp, k, v)
    eye, comp = sim.render(rp)
    oe, oc = O.render(sim.read_density(), rp)
    for got, want in ((eye, oe), (comp, oc)):
        nan = np.isnan(want)  # a NaN's sign and payload are not the restatement's to fix
        assert np.array_equal(np.isnan(got), nan)
        assert np.array_equal(got.view(np.uint32)[~nan], want.view(np.uint32)[~nan])
    sim.close()

"""The FP64 beam kernel's fixed-point parts (rotation matrices, relative rotations, directors, the
moment's rotation) where they take their general forms: quaternions of either sign and any base
orientation, directors that are no unit vectors, moments beyond the exponents a common scale covers,
rotations that are not finite; against the CPU restatement at the bars of the reference fixtures."""
import numpy as np
import pytest
from scipy.spatial.transform import Rotation

from conftest import rel_err
from test_gpu_fp64_paths import model
from test_gpu_objective import TOL

pytestmark = pytest.mark.gpu


def agree(sol, orc, z, top, scale=1.0):
    r, o = sol.objective(z, top, True), orc.objective(z, top, True)
    assert np.isfinite(o["energy"])
    assert abs(r["energy"] - o["energy"]) <= TOL * abs(o["energy"])
    assert rel_err(r["grad"] * scale, o["grad"] * scale) <= TOL
    assert rel_err(r["trial_next"] * scale, o["trial_next"] * scale) <= TOL
    assert np.array_equal(r["trial_flags"], o["trial_flags"])


@pytest.mark.parametrize("sigma_b,sigma_r", [(0.0, 0.1), (0.2, 0.0), (0.5, 0.3), (3.0, 0.5)])
def test_base_orientations_of_either_sign(mcg, mco, sigma_b, sigma_r):
    cfg, lat, sol, orc = model(mcg, mco, "bcc", (3, 2, 2))
    rng = np.random.default_rng(4)
    v = sigma_b * rng.standard_normal((lat.n_nodes, 3))
    a = np.maximum(np.linalg.norm(v, axis=1, keepdims=True), 1e-300)
    q = np.hstack([np.cos(a / 2), np.sin(a / 2) * v / a]) * rng.choice([-1.0, 1.0], (lat.n_nodes, 1))
    z, _ = mcg.random_state(lat, 0.02, sigma_r, 0.0, 5)
    for m in (sol, orc):
        m.set_state(base_r=q.ravel())
    agree(sol, orc, z, lat.geometry.top0 + 0.01)


@pytest.mark.parametrize("length", [1.0, 1.5, 40.0, 1e-3])
def test_directors_that_are_no_unit_vectors(mcg, mco, length):
    cfg, lat, _, _ = model(mcg, mco, "bcc", (2, 2, 2))
    lat.e0[:] = (lat.e0.reshape(-1, 3) * np.where(np.arange(lat.n_beams) % 2, length, 1.0)[:, None]).reshape(lat.e0.shape)
    z, _ = mcg.random_state(lat, 0.02, 0.1, 0.0, 5)
    agree(mcg.Solver(cfg, lat), mco.Model("mco", cfg, lattice=lat), z, lat.geometry.top0 + 0.01)


@pytest.mark.parametrize("young", [2.0e-230, 2.0e-3, 2.0e120])
def test_moments_of_any_exponent(mcg, mco, young):
    cfg, lat, _, _ = model(mcg, mco, "bcc", (2, 2, 2), young=young)
    cfg.material.hardening = 0.05 * young
    cfg.material.yield_ = 1e3 * young  # elastic
    cfg.gravity = cfg.centering_stiffness = cfg.contact_stiffness = 0.0
    z, _ = mcg.random_state(lat, 0.02, 0.1, 0.0, 5)
    agree(mcg.Solver(cfg, lat), mco.Model("mco", cfg, lattice=lat), z, lat.geometry.top0 + 0.01, 1.0 / young)


@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf])
def test_a_rotation_that_is_not_finite(mcg, mco, value):
    cfg, lat, sol, _ = model(mcg, mco, "bcc", (2, 2, 2))
    z, _ = mcg.random_state(lat, 0.02, 0.1, 0.0, 5)
    free = np.flatnonzero(~lat.locked.astype(bool))
    z[free[free % 6 >= 3][7]] = value
    r = sol.objective(z, lat.geometry.top0 + 0.01)
    assert r["energy"] == np.inf and not np.any(r["grad"])


@pytest.mark.parametrize("size", [0.5, 1.9, 2.1, 3.5, 3.9, 4.1, 12.0, 1e6])
def test_plastic_rotations_of_any_size(mcg, mco, size):
    """Plastic rotations along the beams' axes, their largest component of the given size, against
    relative rotations of either direction: the trial twist is larger than any of their components (up to
    sqrt(3) sizes, and pi more or less)."""
    cfg, lat, _, _ = model(mcg, mco, "bcc", (5, 4, 3))
    cfg.material.yield_ = 1e12 * cfg.material.young  # elastic at any of these strains
    sol, orc = mcg.Solver(cfg, lat), mco.Model("mco", cfg, lattice=lat)
    z, _ = mcg.random_state(lat, 0.02, 1.5, 0.0, 5)
    zn = z.reshape(-1, 6)
    x = lat.x0.reshape(-1, 3) + cfg.translation_scale * zn[:, :3]
    R = Rotation.from_rotvec(zn[:, 3:])
    chord = x[lat.beam_b] - x[lat.beam_a]
    axis = R[lat.beam_a].inv().apply(chord / np.linalg.norm(chord, axis=1, keepdims=True))
    sign = np.where(np.arange(lat.n_beams) % 2, 1.0, -1.0)[:, None]
    pl = np.zeros((lat.n_beams, 7))
    pl[:, 2:5] = size * sign * axis / np.max(np.abs(axis), axis=1, keepdims=True)
    twist = np.sum(((R[lat.beam_a].inv() * R[lat.beam_b]).as_rotvec() - pl[:, 2:5]) * axis, axis=1)
    assert np.max(np.abs(twist)) > 1.5 * size
    for m in (sol, orc):
        m.set_state(plastic=pl.ravel())
    agree(sol, orc, z, lat.geometry.top0 + 0.01)
    a, b = (m.objective(z, lat.geometry.top0 + 0.01, True)["trial_aux"].reshape(-1, 7)[:, 2:5] for m in (sol, orc))
    assert rel_err(a, b) <= TOL

@pytest.mark.parametrize("off", [0.0, 1e-12, -1e-9, 1e-8, -1e-7, 5e-7, -5e-7, 9e-7, 1e-3, -0.5])
def test_base_orientations_given_to_few_digits_are_normalized(mcg, mco, off):
    """Base quaternions of length 1 + off: the evaluation's orientations, which a commit keeps, have
    length one to rounding (bar: a squared length by four products and three sums, a square root and a
    quotient, each to half an ulp, 2^-53 relative: 4 of them on a length)."""
    cfg, lat, _, _ = model(mcg, mco, "bcc", (2, 2, 2))
    cfg.max_iterations = 1
    sol = mcg.Solver(cfg, lat)
    rng = np.random.default_rng(8)
    q = rng.standard_normal((lat.n_nodes, 4))
    q /= np.linalg.norm(q, axis=1, keepdims=True)
    sol.set_state(base_r=((1.0 + off) * q).ravel())
    sol.minimize(lat.geometry.top0 + 0.01, np.zeros(6 * lat.n_nodes))
    sol.commit()
    r = sol.get_state()[1].reshape(-1, 4).astype(np.longdouble)
    assert np.max(np.abs(np.sqrt(np.sum(r * r, axis=1)) - 1)) <= 4 * 2.0 ** -53


@pytest.mark.parametrize("value", [np.nan, np.inf, -1e250])
def test_a_plastic_rotation_that_is_not_finite_or_whose_square_is_not(mcg, mco, value):
    cfg, lat, sol, orc = model(mcg, mco, "bcc", (2, 2, 2))
    z, _ = mcg.random_state(lat, 0.02, 0.1, 0.0, 5)
    pl = np.zeros((lat.n_beams, 7))
    pl[17, 3] = value
    for m in (sol, orc):
        m.set_state(plastic=pl.ravel())
    r, o = (m.objective(z, lat.geometry.top0 + 0.01) for m in (sol, orc))
    assert r["energy"] == o["energy"] == np.inf and not np.any(r["grad"]) and not np.any(o["grad"])

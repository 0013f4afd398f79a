"""The FP64 beam kernel's fixed-point parts keep FP64's relative precision at small rotations and
strains: against the CPU restatement at a bar of rounding, not at that of the reference fixtures.

Bars, in units of 2^-53 and of the 2-norm over all beams or nodes.  A moment is a relative rotation
(four products a component), its angle's factor, the projection on the axis and a stiffness, in both
implementations: about a dozen roundings each, 32 together.  A gradient entry adds the transport, the
rotation into the world frame, the shear (its own dozen) and the sum over a node's beams: 64.  The
energy of a state is a sum of squares of the same numbers: 64."""
import numpy as np
import pytest

from conftest import rel_err
from falling_dice_gb300 import abi, workloads

pytestmark = pytest.mark.gpu

U = 2.0 ** -53


def model(mcg, mco, kind, cells, jitter):
    cfg, spec = workloads.bcc(cells, jitter=jitter)
    spec.kind = abi.MCG_LATTICE_CUBIC if kind == "cubic" else abi.MCG_LATTICE_CUBIC_BCC
    cfg.self_contact = 0
    cfg.gravity = cfg.centering_stiffness = 0.0  # the beams alone make energy and gradient
    lat = mcg.generate_lattice(spec, cfg)
    return cfg, lat, mcg.Solver(cfg, lat), mco.Model("mco", cfg, lattice=lat)


def moments(r):
    return r["trial_aux"].reshape(-1, 7)[:, 2:5]


# rotations at the first increment's base state (identity orientations), on struts that lie along
# the axes: every strain is of the rotations' size, and none is a difference of numbers near one
@pytest.mark.parametrize("sigma", [1e-15, 1e-12, 1e-9, 1e-6, 1e-4, 1e-2, 0.1, 0.3, 0.6])
def test_small_rotations_of_an_axis_aligned_lattice(mcg, mco, sigma):
    cfg, lat, sol, orc = model(mcg, mco, "cubic", (5, 4, 3), 0.0)
    z, _ = mcg.random_state(lat, 0.0, sigma, 0.0, 11)
    top = lat.geometry.top0 + 0.01
    r, o = sol.objective(z, top, True), orc.objective(z, top, True)
    assert o["energy"] > 0 and np.any(moments(o))
    assert rel_err(moments(r), moments(o)) <= 32 * U
    assert rel_err(r["grad"], o["grad"]) <= 64 * U
    assert abs(r["energy"] - o["energy"]) <= 64 * U * o["energy"]


# moments keep their digits on struts of any direction, with displacements, from base states that a
# commit left as small rotations, and beside plastic rotations of their own size
@pytest.mark.parametrize("base", [0.0, 1.0])
@pytest.mark.parametrize("plastic", [0.0, 1.0])
@pytest.mark.parametrize("sigma", [1e-12, 1e-9, 1e-6, 1e-3, 0.03])
def test_moments_of_small_rotations(mcg, mco, sigma, plastic, base):
    cfg, lat, sol, orc = model(mcg, mco, "bcc", (4, 3, 3), 0.02)
    z, _ = mcg.random_state(lat, 0.02, sigma, 0.0, 12)
    rng = np.random.default_rng(13)
    v = base * sigma * rng.standard_normal((lat.n_nodes, 3))
    a = np.linalg.norm(v, axis=1, keepdims=True)
    q = np.hstack([np.cos(a / 2), 0.5 * np.sinc(a / (2 * np.pi)) * v])
    pl = np.zeros((lat.n_beams, 7))
    pl[:, 2:5] = plastic * sigma * rng.standard_normal((lat.n_beams, 3))
    for m in (sol, orc):
        m.set_state(base_r=q.ravel(), plastic=pl.ravel())
    top = lat.geometry.top0 + 0.01
    r, o = sol.objective(z, top, True), orc.objective(z, top, True)
    assert np.any(moments(o))
    assert rel_err(moments(r), moments(o)) <= 32 * U
    assert rel_err(r["trial_next"].reshape(-1, 7)[:, 2:5], o["trial_next"].reshape(-1, 7)[:, 2:5]) <= 32 * U


# The chord's length is the correctly rounded square root the reference takes: the residual
# correction leaves an error of the order of 2^-104 before the last rounding.  Strains (L - L0) / L0
# then differ by the quotient's form alone: 1 / L0, a product and a quotient, each to half an ulp.
@pytest.mark.parametrize("scale", [1.0, 1.0 + 1e-12, 1.0 + 1e-7, 0.9, 3.7, 1e-6, 1e9])
def test_chord_lengths_are_the_references(mcg, mco, scale):
    cfg, lat, sol, orc = model(mcg, mco, "bcc", (9, 8, 7), 0.02)
    for m in (sol, orc):
        m.set_state(base_x=lat.x0 * scale)
    z = np.zeros(6 * lat.n_nodes)
    top = 2.0 * scale
    a, b = (m.objective(z, top, True)["trial_aux"].reshape(-1, 7)[:, 0] for m in (sol, orc))
    assert np.all(np.abs(a - b) <= 3 * U * np.abs(b))


# Orientations exp(z) from an identity base, as a commit stores them, against the exponential in
# extended precision: its polynomials' last steps and products, and the normalization, 4 roundings on
# a component (the angles of both the polynomials and the general form, limit one radian).
@pytest.mark.parametrize("sigma", [1e-9, 1e-3, 0.3, 0.6, 1.0, 3.0])
def test_orientations_are_the_exponentials_to_rounding(mcg, mco, sigma):
    cfg, lat, _, _ = model(mcg, mco, "bcc", (4, 3, 3), 0.02)
    cfg.max_iterations = 1
    sol = mcg.Solver(cfg, lat)
    z, _ = mcg.random_state(lat, 0.0, sigma, 0.0, 14)
    z = sol.minimize(lat.geometry.top0 + 0.01, z)[0]
    sol.commit()
    q = sol.get_state()[1].reshape(-1, 4)
    v = z.reshape(-1, 6)[:, 3:].astype(np.longdouble)
    a = np.sqrt(np.sum(v * v, axis=1, keepdims=True))
    s = np.where(a > 0, np.sin(a / 2) / np.where(a > 0, a, 1), np.longdouble(0.5))
    want = np.hstack([np.cos(a / 2), s * v])
    assert np.max(np.abs(q - want)) <= 4 * U

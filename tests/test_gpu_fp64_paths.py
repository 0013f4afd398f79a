"""The FP64 kernels' own evaluations of rotations, lengths and return maps (polynomials up to a
limit and the general functions beyond it, square roots from an FP32 estimate) against the CPU
restatement, at rotations on both sides of every limit and at element counts around the block
sizes.  Bars as in test_gpu_objective.py: 1e-10 relative; the platens stay clear and
self-contact is off, so that the beams alone make the gradient."""
import numpy as np
import pytest

from conftest import rel_err
from falling_dice_gb300 import abi, workloads
from test_gpu_objective import TOL, check_eval, close_cols

pytestmark = pytest.mark.gpu

LATTICES = [("cubic", (1, 1, 1)), ("bcc", (2, 1, 3)), ("bcc", (3, 2, 2)), ("bcc", (5, 4, 3))]  # 12 .. 1023 beams


def model(mcg, mco, kind, cells, young=2.0e9):
    cfg, spec = workloads.bcc(cells, young=young)
    spec.kind = abi.MCG_LATTICE_CUBIC if kind == "cubic" else abi.MCG_LATTICE_CUBIC_BCC
    cfg.self_contact = 0
    lat = mcg.generate_lattice(spec, cfg)
    return cfg, lat, mcg.Solver(cfg, lat), mco.Model("mco", cfg, lattice=lat)


@pytest.mark.parametrize("kind,cells", LATTICES)
@pytest.mark.parametrize("sigma_r", [0.0, 1e-9, 0.05, 0.32, 0.7, 1.6, 3.0])
def test_rotations_on_both_sides_of_the_polynomials(mcg, mco, kind, cells, sigma_r):
    cfg, lat, sol, orc = model(mcg, mco, kind, cells)
    z, _ = mcg.random_state(lat, 0.02, sigma_r, 0.0, 5)
    rng = np.random.default_rng(9)
    pl = np.zeros((lat.n_beams, 7))
    pl[:, :2] = rng.uniform(0, 0.01, (lat.n_beams, 2))
    pl[:, 2:5] = 0.05 * rng.standard_normal((lat.n_beams, 3))
    pl[:, 5:] = rng.uniform(0, 0.05, (lat.n_beams, 2))
    pl[::3] = 0.0
    sol.set_state(plastic=pl.ravel())
    orc.set_state(plastic=pl.ravel())
    top = lat.geometry.top0 + 0.01
    r, o = sol.objective(z, top, True), orc.objective(z, top, True)
    s = {"energy": o["energy"], "grad": o["grad"],
         "diag": np.array([o["diag"][k] for k in ("elastic", "plastic", "contact", "reaction", "max_pen", "contacts")])}
    check_eval(r, s, (kind, cells, sigma_r))
    for k in ("trial_next", "trial_aux"):
        ok, err = close_cols(r[k], o[k], np.zeros(7))
        assert ok, (k, err)
    assert np.array_equal(r["trial_flags"], o["trial_flags"])


def test_chord_lengths_beyond_the_estimates_range(mcg, mco):
    """Positions scaled so that squared chords leave FP32's range: the general square root runs."""
    cfg, lat, sol, orc = model(mcg, mco, "bcc", (2, 2, 1))
    scale = 1e30
    for m in (sol, orc):
        m.set_state(base_x=lat.x0 * scale)
    z = np.zeros(6 * lat.n_nodes)
    r, o = sol.objective(z, 2.0 * scale), orc.objective(z, 2.0 * scale, False)
    assert np.isfinite(o["energy"])
    assert abs(r["energy"] - o["energy"]) <= TOL * abs(o["energy"])
    assert rel_err(r["grad"], o["grad"]) <= TOL


def test_a_nan_position_gives_the_reference_outcome(mcg, mco):
    cfg, lat, sol, orc = model(mcg, mco, "bcc", (2, 2, 2))
    z, _ = mcg.random_state(lat, 0.02, 0.1, 0.0, 5)
    free = np.flatnonzero(~lat.locked.astype(bool))
    z[free[17]] = np.nan
    r = sol.objective(z, lat.geometry.top0 + 0.01)
    assert r["energy"] == np.inf and not np.any(r["grad"])


@pytest.mark.parametrize("cells", [(1, 1, 30), (1, 1, 31), (1, 1, 32), (3, 3, 3), (4, 4, 4), (3, 7, 7), (5, 6, 5)])
def test_node_counts_around_the_block_size(mcg, mco, cells):
    """Cubic lattices of 64 .. 256 nodes (124, 128, 132; blocks of 128 nodes) between both platens
    and with self-contact on: totals, extrema and residual norms of full and partial blocks."""
    cfg, spec = workloads.bcc(cells)
    spec.kind = abi.MCG_LATTICE_CUBIC
    lat = mcg.generate_lattice(spec, cfg)
    sol, orc = mcg.Solver(cfg, lat), mco.Model("mco", cfg, lattice=lat)
    z, pl = mcg.random_state(lat, 0.2, 0.1, 0.02, 21)
    for m in (sol, orc):
        m.set_state(plastic=pl)
    top = lat.geometry.top0 - 0.1 * lat.geometry.height
    r, o = sol.objective(z, top), orc.objective(z, top, False)
    s = {"energy": o["energy"], "grad": o["grad"],
         "diag": np.array([o["diag"][k] for k in ("elastic", "plastic", "contact", "reaction", "max_pen", "contacts")])}
    check_eval(r, s, cells)
    assert np.array_equal(sol.contact_pairs(), orc.contact_pairs(z))

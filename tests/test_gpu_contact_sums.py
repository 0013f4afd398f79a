"""Contact forces and energies as fixed-point sums (quantum 2^-90 below stiffness times a
reference length of the configuration): lattices whose lengths and stiffness lie far from the
reference's, and stiffnesses that are zero or not finite, against the CPU restatement.  Bars as in
test_gpu_objective.py: a sum is exact and rounded once, so 1e-10 holds wherever FP64 resolves the
penetrations themselves."""
import numpy as np
import pytest

from conftest import rel_err
from falling_dice_gb300 import workloads
from test_gpu_objective import TOL, check_eval

pytestmark = pytest.mark.gpu


def squeezed_pair(mcg, mco, scale=1.0, **kw):
    """A 5x5x4 cubic+BCC lattice of cells `scale` times 5 mm squeezed to half its height."""
    cfg, spec = workloads.bcc((5, 5, 4), r0=0.4e-3 * scale, r1=0.7e-3 * scale)
    cfg.cell_size *= scale
    cfg.min_radius, cfg.max_radius = 0.4e-3 * scale, 0.7e-3 * scale
    cfg.contact_margin *= scale
    cfg.translation_scale = cfg.cell_size
    spec.cell_size = cfg.cell_size
    for k, v in kw.items():
        setattr(cfg, k, v)
    lat = mcg.generate_lattice(spec, cfg)
    z, pl = mcg.random_state(lat, 0.2, 0.1, 0.02, 77)
    y = lat.x0[1::3]
    z[1::6] -= 0.5 * (y - y.min()) / cfg.translation_scale
    z[lat.locked.astype(bool)] = 0
    top = lat.geometry.top0 - 0.5 * lat.geometry.height
    sol, orc = mcg.Solver(cfg, lat), mco.Model("mco", cfg, lattice=lat)
    for m in (sol, orc):
        m.set_state(plastic=pl)
    o = orc.objective(z, top, False)
    return sol, sol.objective(z, top), o, orc.contact_pairs(z)


@pytest.mark.parametrize("scale", [1e-6, 1e-3, 1.0, 1e4])
@pytest.mark.parametrize("stiffness", [1e-30, 1.2e6, 1e60])
def test_contact_sums_at_any_scale(mcg, mco, scale, stiffness):
    sol, r, o, pairs = squeezed_pair(mcg, mco, scale, contact_stiffness=stiffness)
    assert len(pairs) > 200 and np.array_equal(sol.contact_pairs(), pairs)
    d, ref = r["diag"], o["diag"]
    assert d["contacts"] == ref["contacts"] and d["max_pen"] == ref["max_pen"]
    assert abs(d["contact"] - ref["contact"]) <= TOL * ref["contact"]
    assert abs(r["energy"] - o["energy"]) <= TOL * abs(o["energy"])
    assert rel_err(r["grad"], o["grad"]) <= TOL
    again = sol.objective(*sol_args(sol))
    assert again["energy"] == r["energy"] and np.array_equal(again["grad"], r["grad"])  # the sums were cleared


def sol_args(sol):
    """The state squeezed_pair evaluates (the generator is seeded)."""
    lat, cfg = sol.lattice, sol.cfg
    import falling_dice_gb300 as fd
    z, _ = fd.random_state(lat, 0.2, 0.1, 0.02, 77)
    y = lat.x0[1::3]
    z[1::6] -= 0.5 * (y - y.min()) / cfg.translation_scale
    z[lat.locked.astype(bool)] = 0
    return z, lat.geometry.top0 - 0.5 * lat.geometry.height


def test_zero_stiffness_leaves_only_the_count(mcg, mco):
    sol, r, o, pairs = squeezed_pair(mcg, mco, contact_stiffness=0.0)
    s = {"energy": o["energy"], "grad": o["grad"],
         "diag": np.array([o["diag"][k] for k in ("elastic", "plastic", "contact", "reaction", "max_pen", "contacts")])}
    check_eval(r, s, "zero stiffness")
    assert np.array_equal(sol.contact_pairs(), pairs)


@pytest.mark.parametrize("stiffness", [np.inf, np.nan])
def test_a_stiffness_that_is_not_finite_gives_the_non_finite_outcome(mcg, mco, stiffness):
    sol, r, o, _ = squeezed_pair(mcg, mco, contact_stiffness=stiffness)
    assert o["energy"] == np.inf and not np.any(o["grad"])
    assert r["energy"] == np.inf and not np.any(r["grad"])


def test_an_overflow_seen_while_the_first_lattice_rests(mcg):
    """Contact buffers that overflow in a batch's run after its first lattice has finished: the
    evaluation is repeated with larger buffers all the same, so the runs are those of ample ones."""
    cfg, _ = workloads.bcc((3, 3, 3), contact_stiffness=workloads.CONTACT_STIFF)
    cfg.load_steps, cfg.unload_steps, cfg.max_strain = 2, 0, 0.05
    lats = []
    for n, seed in ((2, 5), (4, 6), (5, 7)):
        _, spec = workloads.bcc((n, n, n), 0.3e-3, 0.5e-3, 0.03)
        spec.seed = seed
        lats.append(mcg.generate_lattice(spec, cfg))
    runs = []
    for small in (False, True):
        b = mcg.BatchSolver(cfg, lats)
        if small:
            b.set_contact_capacity(8, 4096, 4096, 4096)
        status, frames = b.run()
        runs.append((list(status), frames))
        b.close()
    assert runs[0] == runs[1]

"""The node gather and the totals at the sizes where their blocks and paths end: fewer nodes than a
64-node gather block, exactly one and two, one more; and lattices on either side of the number of
block partials (768) up to which the last gather block sums the totals instead of a kernel of its
own.  FP64 against the CPU restatement at the bars of the reference fixtures; both forms in a batch,
bit for bit what each lattice gives alone."""
import numpy as np
import pytest

from conftest import rel_err
from falling_dice_gb300 import abi, workloads

pytestmark = pytest.mark.gpu


def specimen(mcg, cells, kind, precision=abi.MCG_FP64):
    cfg, spec = workloads.bcc(cells)
    spec.kind = kind
    cfg.precision = precision
    lat = mcg.generate_lattice(spec, cfg)
    z, pl = mcg.random_state(lat, 0.05, 0.1, 0.02, 7)
    return cfg, lat, z, pl, lat.geometry.top0 - 0.002


# nodes: 8, 63, 64, 66, 126, 128, 130; 2048 and 2057 (the gradient's two ways to the host)
SMALL = [(1, 1, 1), (2, 2, 6), (3, 3, 3), (1, 2, 10), (2, 5, 6), (1, 7, 7), (1, 4, 12), (15, 15, 7), (10, 10, 16)]
# block partials of the cubic+BCC lattices: 717 and 841
CASES = [(c, abi.MCG_LATTICE_CUBIC) for c in SMALL] + [((n, n, n), abi.MCG_LATTICE_CUBIC_BCC) for n in (18, 19)]


@pytest.mark.parametrize("cells,kind", CASES)
def test_totals_and_gradient_against_the_restatement(mcg, mco, cells, kind):
    cfg, lat, z, pl, top = specimen(mcg, cells, kind)
    sol, orc = mcg.Solver(cfg, lat), mco.Model("mco", cfg, lattice=lat)
    sol.set_state(plastic=pl)
    orc.set_state(plastic=pl)
    r, o = sol.objective(z, top), orc.objective(z, top)
    assert abs(r["energy"] - o["energy"]) <= 1e-10 * abs(o["energy"])
    assert rel_err(r["grad"], o["grad"]) <= 1e-10
    for k in ("elastic", "plastic", "contact", "reaction"):
        assert abs(r["diag"][k] - o["diag"][k]) <= 1e-10 * max(abs(o["diag"][k]), 1e-12), k
    assert r["diag"]["max_pen"] == o["diag"]["max_pen"] and r["diag"]["contacts"] == int(o["diag"]["contacts"])


# beams: 2048 and 2049 (the trial states' two ways to the host); cubic (a, b, c)
@pytest.mark.parametrize("cells", [(7, 7, 11), (2, 9, 26)])
@pytest.mark.parametrize("precision", [abi.MCG_FP64, abi.MCG_MIXED])
def test_what_the_host_receives_is_what_the_device_holds(mcg, precision, cells):
    cfg, lat, z, pl, top = specimen(mcg, cells, abi.MCG_LATTICE_CUBIC, precision)
    sol = mcg.Solver(cfg, lat)
    sol.set_state(plastic=pl)
    a = sol.objective(z, top, True)
    b = sol.objective(z, top)
    c = sol.read_result()
    assert a["energy"] == b["energy"] == c["energy"]
    assert np.array_equal(a["grad"], b["grad"]) and np.array_equal(a["grad"], c["grad"])
    for k in ("trial_next", "trial_aux"):
        assert np.all(np.isfinite(a[k])) and np.any(a[k])
    # a state that is not finite: no gradient anywhere; then the same state again
    bad = z.copy()
    bad[np.flatnonzero(~lat.locked.astype(bool))[5]] = np.nan
    r = sol.objective(bad, top, True)
    assert r["energy"] == np.inf and not np.any(r["grad"]) and not np.any(sol.read_result()["grad"])
    d = sol.objective(z, top, True)
    assert np.array_equal(a["grad"], d["grad"])
    for k in ("trial_next", "trial_aux", "trial_flags"):
        assert np.array_equal(a[k], d[k])


@pytest.mark.parametrize("precision,sizes", [(abi.MCG_FP64, (19, 1, 18, 3)), (abi.MCG_MIXED, (22, 1, 21, 3))])
def test_a_batch_across_the_paths_is_bitwise_the_single_lattices(mcg, precision, sizes):
    parts = [specimen(mcg, (n, n, n), abi.MCG_LATTICE_CUBIC_BCC, precision) for n in sizes]
    batch = mcg.BatchSolver(parts[0][0], [p[1] for p in parts])
    batch.set_state(plastic=np.concatenate([p[3] for p in parts]))
    got = batch.objective(np.concatenate([p[2] for p in parts]), [p[4] for p in parts])
    off = batch.node_offsets
    for k, (cfg, lat, z, pl, top) in enumerate(parts):
        sol = mcg.Solver(cfg, lat)
        sol.set_state(plastic=pl)
        ref = sol.objective(z, top)
        assert got["energy"][k] == ref["energy"], k
        assert np.array_equal(got["grad"][6 * off[k]:6 * off[k + 1]], ref["grad"]), k
        assert got["diag"][k] == ref["diag"], k


@pytest.mark.parametrize("precision", [abi.MCG_FP64, abi.MCG_MIXED])
def test_a_gradient_copied_in_pieces_is_the_device_s(mcg, precision):
    """205,379 nodes (copied while it is gathered), alone and behind a small lattice in a batch whose
    large or small lattice is not finite: every call returns its own state's gradient."""
    cfg, lat, z, pl, top = specimen(mcg, (58, 58, 58), abi.MCG_LATTICE_CUBIC, precision)
    sol = mcg.Solver(cfg, lat)
    sol.set_state(plastic=pl)
    want = {}
    for s in (1.0, 0.5):
        sol.upload_z(s * z)
        sol.objective_resident(top)
        want[s] = sol.read_result()
    for k in range(12):
        s = 1.0 if k % 3 else 0.5
        r = sol.objective(s * z, top)
        assert r["energy"] == want[s]["energy"] and np.array_equal(r["grad"], want[s]["grad"]), k
    _, small, zs, ps, _ = specimen(mcg, (3, 3, 3), abi.MCG_LATTICE_CUBIC, precision)
    batch = mcg.BatchSolver(cfg, [small, lat])
    batch.set_state(plastic=np.concatenate([ps, pl]))
    tops = [small.geometry.top0, top]
    for bad in (None, 0, 1):
        zz = [zs.copy(), z.copy()]
        if bad is not None:
            one = (small, lat)[bad]
            zz[bad][np.flatnonzero(~one.locked.astype(bool))[4]] = np.nan
        r = batch.objective(np.concatenate(zz), tops)
        g = np.split(r["grad"], [6 * small.n_nodes])
        assert np.array_equal(g[1], want[1.0]["grad"]) if bad != 1 else not np.any(g[1])
        assert np.any(g[0]) == (bad != 0)

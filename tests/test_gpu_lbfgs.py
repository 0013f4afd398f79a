"""The search directions at the sizes where the solver's blocks and register arrays end: lattices
of less than a 64-node block, exactly one, one and a bit, all 152 blocks and just more (longer
runs of nodes per block); histories around the pairs a block takes (4), a thread's registers (12),
the shared-memory solve (16), a warp (32) and the largest (64), each over more iterations than it
holds, against the CPU restatement's minimize.

Bars: the same iteration count; a 1e-12 perturbation of the restatement's start changes its
result by at most 1e-8 in z and 5e-11 in energy after 40 iterations, and 7e-6 and 3e-9 after 72;
allowed is a hundred times that.
"""
import numpy as np
import pytest

from conftest import rel_err
from falling_dice_gb300 import abi, workloads

pytestmark = pytest.mark.gpu


def specimen(mcg, cells, history, iterations):
    cfg, spec = workloads.bcc(cells)
    spec.kind = abi.MCG_LATTICE_CUBIC
    cfg.history, cfg.max_iterations, cfg.relative_gradient_tolerance = history, iterations, 1e-8
    lat = mcg.generate_lattice(spec, cfg)
    return cfg, lat, lat.geometry.top0 - 0.08 * lat.geometry.height


def check(mcg, mco, cells, history, iterations):
    cfg, lat, top = specimen(mcg, cells, history, iterations)
    z0 = np.zeros(6 * lat.n_nodes)
    zo, so, eo, _ = mco.Model("mco", cfg, lattice=lat).minimize(top, z0)
    z, s, e, _ = mcg.Solver(cfg, lat).minimize(top, z0)
    assert s["iterations"] == so["iterations"]
    tz, te = (1e-6, 5e-9) if iterations <= 40 else (7e-4, 3e-7)
    assert rel_err(z, zo) <= tz, rel_err(z, zo)
    assert abs(e - eo) <= te * abs(eo), (e, eo)


# nodes: 8, 64, 66, 125
@pytest.mark.parametrize("cells", [(1, 1, 1), (3, 3, 3), (1, 2, 10), (4, 4, 4)])
@pytest.mark.parametrize("history,iterations", [(1, 8), (4, 12), (5, 14), (8, 20), (10, 24), (12, 28), (13, 30),
                                                (16, 36), (17, 40), (33, 72), (64, 72)])
def test_directions_for_histories_of_any_length(mcg, mco, cells, history, iterations):
    if cells == (1, 1, 1):
        iterations = min(iterations, 7)  # the frame of eight nodes reaches its minimum to rounding
    check(mcg, mco, cells, history, iterations)


# nodes: 9728 = 152 blocks of 64, 9747: blocks of 128
@pytest.mark.parametrize("cells", [(15, 31, 18), (18, 18, 26)])
@pytest.mark.parametrize("history", [5, 13])
def test_directions_where_the_blocks_run_out(mcg, mco, cells, history):
    check(mcg, mco, cells, history, 12)


def test_a_batch_of_these_sizes_is_bitwise_the_single_runs(mcg):
    sizes = [(18, 18, 26), (1, 1, 1), (3, 3, 3), (15, 31, 18), (1, 2, 10)]
    cfg, _, _ = specimen(mcg, sizes[0], 10, 30)
    cfg.load_steps, cfg.unload_steps, cfg.max_strain = 2, 0, 0.02
    lats = [specimen(mcg, c, 10, 30)[1] for c in sizes]
    status, runs = mcg.BatchSolver(cfg, lats).run()
    for k, lat in enumerate(lats):
        rc, ref = mcg.Solver(cfg, lat).run()
        assert status[k] == rc and runs[k] == ref, k

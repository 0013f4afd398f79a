"""The pair enumeration at the sizes where its blocks end: bins of 1 to several hundred shapes
(groups of 32, chunks of 128, several chunks) and cells from a fraction of a strut to the whole
specimen, against the CPU restatement's contact pair set."""
import numpy as np
import pytest

from falling_dice_gb300 import abi, workloads

pytestmark = pytest.mark.gpu


def squeezed(mcg, kind, cells, share, sigma):
    cfg, spec = workloads.bcc(cells, r0=0.5e-3, r1=0.9e-3)
    spec.kind = kind
    lat = mcg.generate_lattice(spec, cfg)
    z, pl = mcg.random_state(lat, sigma, 0.1, 0.02, 31)
    y = lat.x0[1::3]
    z[1::6] -= share * (y - y.min()) / cfg.translation_scale
    z[lat.locked.astype(bool)] = 0
    return cfg, lat, z


# shapes (nodes + beams): 20, 33, 54, 81, 72, 128, 158, 386, 700
SIZES = [(abi.MCG_LATTICE_CUBIC, (1, 1, 1)), (abi.MCG_LATTICE_CUBIC, (2, 1, 1)), (abi.MCG_LATTICE_CUBIC, (2, 2, 1)),
         (abi.MCG_LATTICE_CUBIC, (2, 2, 2)), (abi.MCG_LATTICE_CUBIC_BCC, (2, 1, 1)),
         (abi.MCG_LATTICE_CUBIC, (3, 3, 2)), (abi.MCG_LATTICE_CUBIC_BCC, (2, 2, 2)),
         (abi.MCG_LATTICE_CUBIC_BCC, (3, 3, 3)), (abi.MCG_LATTICE_CUBIC_BCC, (4, 4, 3))]


@pytest.mark.parametrize("kind,cells", SIZES)
@pytest.mark.parametrize("cell", [0.0, 1.1e-3, 4e-3, 9e-3, 1.0])
def test_pair_sets_for_bins_of_any_size(mcg, mco, kind, cells, cell):
    cfg, lat, z = squeezed(mcg, kind, cells, 0.55, 0.3)
    sol, orc = mcg.Solver(cfg, lat), mco.Model("mco", cfg, lattice=lat)
    sol.set_contact_cell(cell)
    sol.objective(z, lat.geometry.top0)
    pairs = orc.contact_pairs(z)
    assert np.array_equal(sol.contact_pairs(), pairs)
    st = sol.contact_stats()
    if cell == 1.0:  # every shape in one bin (or the few around the origin's corner)
        assert st["entries"] >= lat.n_nodes + lat.n_beams
    # the candidates hold every contact, and no pair twice
    assert st["filtered"] <= st["candidates"] and st["contacts"] == len(pairs)

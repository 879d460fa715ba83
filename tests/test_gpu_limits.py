"""Calls at their limits: rows of the neighbour list at the capacity and beyond what a warp stages."""
import numpy as np
import pytest

import oracle_binding as ob
from protocell_genesis_b200 import _abi, config as cfgm
from protocell_genesis_b200.soup import SoupSystem

pytestmark = pytest.mark.gpu
P = cfgm.load_params()


def _edge_lattice(capacity, widen=2e-6):
    """a cubic lattice of the list range / sqrt(41), widened so that the 96 neighbours at the range lie just beyond
    it, where the exact distance decides: an inner bead has 1044 neighbours in range"""
    opts = cfgm.SoupOptions(box=[18] * 3, seed=1, kT=1.1, start={"C": 0, "O": 0, "H": 0, "M": 1, "W": 17 ** 3 - 1},
                            verlet_override={"listCapacity": capacity})
    cfg = cfgm.resolve(opts, P)
    a = cfg.list_range / np.sqrt(41.0) * (1.0 + widen)
    assert 16 * a < 18 - cfg.list_range                  # no pair across the faces
    pos = ob.OracleSystem(_abi, cfg).read(ob.F_POS).reshape(-1, 4).copy()
    pos[:, :3] = np.stack(np.meshgrid(*[np.arange(17)] * 3, indexing="ij"), -1).reshape(-1, 3) * a + 0.25
    return cfg, pos.astype(np.float32).ravel()


@pytest.mark.parametrize("capacity", [1044, 1048, 1112, 1136, 1144])
def test_rows_cut_by_candidates_on_the_edge_of_the_range(capacity):
    """rows of 1044 entries, and 96 candidates that the exact distance leaves out: they fit every capacity here"""
    cfg, pos = _edge_lattice(capacity)
    o, g = ob.OracleSystem(_abi, cfg, {"positions": pos}), SoupSystem(cfg, {"positions": pos})
    oc, ol = o.verlet()
    gc, gl = g.verlet_lists()
    assert oc.max() == 1044
    assert np.array_equal(gc, oc)
    assert np.array_equal(gl, ol)
    g.dispose()


def test_rows_beyond_the_capacity_are_reported():
    """a capacity of 1040 holds neither all of the 1044 neighbours nor more than 1040 of them"""
    cfg, pos = _edge_lattice(1040)
    g = SoupSystem(cfg, {"positions": pos})
    counts, _ = g.verlet_lists()
    assert counts.max() == 1040
    with pytest.raises(_abi.SoupError, match="listCapacity"):
        g.relax_cold_start(1, 1e-6)
    g.dispose()

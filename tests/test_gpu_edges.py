"""Kernels at the edges of their tiles and of their dispatch rules, against the CPU oracle or one another:
list builds (grids cut finer along x or not, an axis visited whole, rows longer than a warp's chunks, pairs on the edge of
the list range), the list force's lanes per bead, the far force's rows around its unroll, bond components that go through the
rounds, aggregates on few cells, the flood on odd grids, and the state behind a differentiable window."""
import numpy as np
import pytest

import oracle_binding as ob
from helpers import boosted, charged_opts, plain_opts, rel_rms
from protocell_genesis_b200 import _abi, config as cfgm
from protocell_genesis_b200.soup import SoupSystem
from test_gpu_parity import FORCE_TOL, make_pair, oracle_state
from test_oracle_pins import SYN_BOX, ST, _assemble, _shell, _water

pytestmark = pytest.mark.gpu
P = cfgm.load_params()


def _lists_equal(o, g):
    gc, gl = g.verlet_lists()
    oc, ol = o.verlet()
    assert np.array_equal(gc, oc)
    assert np.array_equal(gl, ol)
    return gc


@pytest.mark.parametrize("box", [[15, 15, 15], [15, 22.3, 31], [40, 15, 15], [60, 60, 60], [17.7, 16.1, 48.9]])
@pytest.mark.parametrize("n", [31, 400, 2600])
def test_lists_over_grids(box, n):
    """dense boxes cut x finer, sparse ones do not (60^3 holds more cells than beads)"""
    opts = cfgm.SoupOptions(box=box, seed=n, kT=1.1, start={"C": 0, "O": 0, "H": 0, "M": 1, "W": n - 1},
                            verlet_override={"listCapacity": 1024})
    cfg = cfgm.resolve(opts, P)
    rng = np.random.default_rng(n)
    pos = ob.OracleSystem(_abi, cfg).read(ob.F_POS).reshape(-1, 4).copy()
    pos[:, :3] = rng.random((cfg.n, 3)) * np.array(box)
    pos[:3, :3] = [[0, 0, 0], [np.nextafter(np.float32(box[0]), np.float32(0)), 0, 0], np.array(box) / 2]
    pos = pos.astype(np.float32).ravel()
    o, g = ob.OracleSystem(_abi, cfg, {"positions": pos}), SoupSystem(cfg, {"positions": pos})
    _lists_equal(o, g)
    g.dispose()


@pytest.mark.parametrize("cells", [(16, 16, 16), (17, 16, 16), (163, 161, 161)])
def test_lists_over_the_scans_of_their_cells(cells):
    """4096 cells are scanned in one launch, up to 1024 blocks of them in two, more by a scan of the blocks' totals"""
    def opts(box):
        return cfgm.SoupOptions(box=box, seed=5, kT=1.1, start={"C": 0, "O": 0, "H": 0, "M": 1, "W": 799})
    half = cfgm.resolve(opts([30.0] * 3), P).list_range / 2
    cfg = cfgm.resolve(opts([(c + 0.3) * half for c in cells]), P)
    box = np.array(cells) * half + 0.3 * half
    rng = np.random.default_rng(5)
    pos = ob.OracleSystem(_abi, cfg).read(ob.F_POS).reshape(-1, 4).copy()
    at = rng.random((200, 3)) * box                      # clumps of four all over the box
    at[:2] = [0.0, 0.0, 0.0], box - 0.5
    pos[:, :3] = np.mod(np.repeat(at, 4, axis=0) + rng.normal(size=(800, 3)), box)
    pos = pos.astype(np.float32).ravel()
    o, g = ob.OracleSystem(_abi, cfg, {"positions": pos}), SoupSystem(cfg, {"positions": pos})
    assert _lists_equal(o, g).max() >= 3
    g.dispose()


@pytest.mark.parametrize("n", [17, 33, 513, 700])
def test_rows_of_any_length(n):
    """every bead in range of every other one: rows of n - 1 entries"""
    opts = cfgm.SoupOptions(box=[20] * 3, seed=1, kT=1.1, start={"C": 0, "O": 0, "H": 0, "M": 1, "W": n - 1},
                            verlet_override={"listCapacity": 1000})
    cfg = cfgm.resolve(opts, P)
    pos = ob.OracleSystem(_abi, cfg).read(ob.F_POS).reshape(-1, 4).copy()
    pos[:, :3] = np.random.default_rng(n).random((n, 3)) * 1.6 + 19.0
    pos[:, :3] %= 20.0
    pos = pos.astype(np.float32).ravel()
    o, g = ob.OracleSystem(_abi, cfg, {"positions": pos}), SoupSystem(cfg, {"positions": pos})
    assert _lists_equal(o, g).min() == n - 1
    g.dispose()


def test_pairs_on_the_edge_of_the_range():
    """a lattice of a third of the list range: dozens of pairs a bead lie within rounding of the range"""
    opts = cfgm.SoupOptions(box=[18] * 3, seed=1, kT=1.1, start={"C": 0, "O": 0, "H": 0, "M": 1, "W": 999},
                            verlet_override={"listCapacity": 600})
    cfg = cfgm.resolve(opts, P)
    a = cfg.list_range / 3
    pos = ob.OracleSystem(_abi, cfg).read(ob.F_POS).reshape(-1, 4).copy()
    at = np.stack(np.meshgrid(*[np.arange(10)] * 3, indexing="ij"), -1).reshape(-1, 3)
    pos[:, :3] = at * a
    pos[:, :3] %= 18.0
    pos = pos.astype(np.float32).ravel()
    o, g = ob.OracleSystem(_abi, cfg, {"positions": pos}), SoupSystem(cfg, {"positions": pos})
    _lists_equal(o, g)
    g.dispose()


def test_lanes_per_bead_change_no_bit(monkeypatch):
    cfg, o, g0 = make_pair(charged_opts(), relax=20)
    g0.dispose()
    runs = []
    for lanes in ("4", "8", "16"):
        monkeypatch.setenv("SOUP_TPP", lanes)
        g = SoupSystem(cfg, oracle_state(o))
        first = g.forces_no_rebuild()
        g.step(25)
        runs.append((first, g.particles(), g.velocities(), g.forces_no_rebuild(), g.charges()))
        g.dispose()
    for other in runs[1:]:
        for a, b in zip(runs[0], other):
            assert np.array_equal(a, b)


@pytest.mark.parametrize("heads", [2, 32, 33, 34, 129, 130, 257])
def test_far_force_rows_around_the_unroll(heads):
    """every head in the far list of every other one: rows of heads - 1 entries"""
    opts = cfgm.SoupOptions(box=[20] * 3, seed=heads, kT=1.1, start={"C": 0, "O": heads, "H": 0, "M": 1, "W": 500},
                            electrostatics={"enabled": True, "pH": 9.0, "ionicStrengthMolar": 0.01})
    cfg = cfgm.resolve(opts, P)
    cfg.es_list_capacity = 512
    o = ob.OracleSystem(_abi, cfg)
    o.relax(20, 0.1)
    g = SoupSystem(cfg, oracle_state(o))
    assert rel_rms(g.forces(), o.forces64()) < FORCE_TOL
    g.dispose()


@pytest.mark.parametrize("box", [10.5, 13.0])
def test_bond_components_in_rounds(box):
    """reactive beads packed closely: components of many items, and single ones, in one pass"""
    def tw(c):
        boosted(c, attempt=1.0, accept=1.0, brk=0.3)
        c.max_hold_steps = 40
    opts = plain_opts(box=[15, 15, box + 5], start={"C": 1500, "O": 300, "H": 0, "M": 250, "W": 0})
    cfg, o, g = make_pair(opts, relax=30, tweak=tw)
    for rnd in range(4):
        o.step(7)
        g.write_state(oracle_state(o))
        o.phase(_abi.PHASE_REBUILD)
        o.phase(_abi.PHASE_BONDS)
        g.debug_phase(_abi.PHASE_BONDS)
        assert np.array_equal(g.bond_slots(), o.read(ob.F_SLOTS)), rnd
        assert np.array_equal(g.center_links(), o.read(ob.F_CENTER)), rnd
        assert np.array_equal(g.center_held_steps(), o.read(ob.F_HELD)), rnd
        assert np.array_equal(g.events_raw(), o.read(ob.F_EVENTS)), rnd
    assert o.read(ob.F_EVENTS).sum() > 100
    g.dispose()


@pytest.mark.parametrize("cutoff", [1.3, 4.0, 6.4, 7.4])
def test_aggregates_on_few_cells(cutoff):
    """11, 3, 2 and 2 cells an axis; thinned members, so that more than one component is left"""
    opts = plain_opts(box=[15] * 3, start={"C": 300, "O": 0, "H": 0, "M": 1, "W": 0})
    cfg = cfgm.resolve(opts, P)
    pos = ob.OracleSystem(_abi, cfg).read(ob.F_POS)
    g = SoupSystem(cfg, {"positions": pos})
    members = np.arange(0, cfg.n, 29 if cutoff > 3 else 2, dtype=np.uint32)
    n_o, lab_o = ob.aggregates(_abi, pos, members, cfg.box, cutoff)
    n_g, lab_g = g.aggregate_labels(members, cutoff)
    assert n_g == n_o and np.array_equal(lab_g, lab_o)
    g.dispose()


@pytest.mark.parametrize("cell", [0.37, 0.5, 0.83, 1.9])
def test_flood_on_odd_grids(cell):
    rng = np.random.default_rng(7)
    centre = np.array([25.0, 25.0, 25.0])
    pos, mem, wat = _assemble(_shell(rng, centre), _water(rng, centre, 500, 3000))
    n = len(pos) // 4
    opts = cfgm.SoupOptions(box=SYN_BOX, seed=1, kT=1.1, start={"C": len(mem), "O": 0, "H": 0, "M": 0, "W": n - len(mem)},
                            verlet_override={"listCapacity": 4096})
    g = SoupSystem(cfgm.resolve(opts, P), {"positions": pos})
    c = ob.periodic_centre(_abi, pos, mem, SYN_BOX, P["circularAlpha"])
    ro = ob.closure(_abi, pos, mem, wat, SYN_BOX, c, cell, ST["closureRadius"], ST["enclosedVolume"])
    rg = g.closure(mem, wat, c, cell, ST["closureRadius"], ST["enclosedVolume"])
    assert rg["encapsulatedCount"] == ro.encapsulated_count and rg["seedCell"] == ro.seed_cell
    assert rg["totalEmptyCells"] == ro.total_empty_cells and rg["unreachedCells"] == ro.unreached_cells
    g.dispose()


def test_a_window_leaves_its_end_behind():
    """the reverse pass puts the window's end back, whatever was done to the system since"""
    import torch
    cfg, o, g = make_pair(charged_opts(rebuild_on_drift=True, skin=1.0), relax=20)
    traj = torch.empty((19, cfg.n, 4), device="cuda")
    torch.cuda.synchronize()
    g.diff_forward(18, 6, traj.data_ptr())

    def state():
        r = g.rng_state()
        return [g.particles(), g.velocities(), g.charges(), g.bond_slots(), g.center_links(), r["bond"], r["thermo"]]
    want = state()
    assert np.array_equal(want[0].reshape(-1, 4), traj[-1].cpu().numpy())
    g.step(30)                                # bonds, charges and velocities move on
    dldx = torch.ones((19, cfg.n, 4), device="cuda")
    torch.cuda.synchronize()
    g.diff_backward(dldx.data_ptr())
    for a, b in zip(want, state()):
        assert np.array_equal(a, b)
    g.step(1)
    g.dispose()


def test_a_sweep_keeps_the_lists_while_they_serve():
    cfg, o, g = make_pair(charged_opts(rebuild_on_drift=True, skin=0.6), relax=20)
    g.step(3)

    def force_is_right():
        now = ob.OracleSystem(_abi, cfg, dict(positions=g.particles(), charges=g.charges(), bond_slots=g.bond_slots(),
                                              center_link=g.center_links()))
        return rel_rms(g.forces_no_rebuild(), now.forces64()) < FORCE_TOL
    built = g.info()["rebuilds"]
    g.debug_phase(_abi.PHASE_MAX_DRIFT)
    g.protonation_sweep()
    assert g.info()["rebuilds"] == built and force_is_right()
    for _ in range(100):                      # kicks and drifts alone: no step looks at the drift
        for _ in range(5):
            g.debug_phase(_abi.PHASE_KICK_DRIFT)
        g.protonation_sweep()
        if g.info()["rebuilds"] > built:
            break
    assert g.info()["rebuilds"] == built + 1 and force_is_right()
    g.dispose()

"""Calls at their limits and calls between others: rows of the neighbour list at the capacity and beyond what a warp
stages, rebuilds of a box of many more cells than beads, a window's reverse pass behind other calls, a sweep on lists
that no longer serve, one in a box below twice its cutoff, aggregates of coordinates far outside the box, the lanes of
the list force, and the sweep's arrays in live boxes and many replicas."""
import numpy as np
import pytest

import oracle_binding as ob
from helpers import charged_opts, confined_opts, oracle_bilayer_start, rel_rms
from protocell_genesis_b200 import _abi, config as cfgm
from protocell_genesis_b200.soup import SoupBatch, SoupSystem
from test_gpu_parity import FORCE_TOL, make_pair, oracle_state

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


@pytest.mark.parametrize("n", [1279, 1280, 1281, 1282, 1297, 2000, 4999])
def test_rows_longer_than_a_staged_row(n):
    """a clump in which every bead is in range of every other: rows of n - 1 entries, of which 1280 are staged; a few
    beads outside it keep ordinary rows"""
    opts = cfgm.SoupOptions(box=[20] * 3, seed=1, kT=1.1, start={"C": 0, "O": 0, "H": 0, "M": 1, "W": n + 9},
                            verlet_override={"listCapacity": 8192})
    cfg = cfgm.resolve(opts, P)
    pos = ob.OracleSystem(_abi, cfg).read(ob.F_POS).reshape(-1, 4).copy()
    pos[:, :3] = np.random.default_rng(n).random((n + 10, 3)) * 1.6 + 19.0
    pos[n:, :3] = 10.0 + 0.5 * np.arange(10)[:, None]
    pos[:, :3] %= 20.0
    pos = pos.astype(np.float32).ravel()
    o, g = ob.OracleSystem(_abi, cfg, {"positions": pos}), SoupSystem(cfg, {"positions": pos})
    oc, ol = o.verlet()
    gc, gl = g.verlet_lists()
    assert oc[:n].min() >= n - 1 and oc[n:].max() < 1280
    assert np.array_equal(gc, oc)
    assert np.array_equal(gl, ol)
    g.dispose()


def test_shells_of_rows_longer_than_a_staged_row(monkeypatch):
    """a dense slab (rows of 1400 entries and more) whose inner beads move: the force read to the drift's shell is the
    force over the whole rows, bit for bit, and the one over every pair"""
    a, cells = 0.62, (25, 25, 15)
    box = [25 * a, 25 * a, 40.0]
    n = int(np.prod(cells))
    opts = cfgm.SoupOptions(box=box, seed=1, kT=1.1, start={"C": 0, "O": 0, "H": 0, "M": 1, "W": n - 1},
                            verlet_override={"listCapacity": 2048})
    cfg = cfgm.resolve(opts, P)
    cfg.dt = 1e-6                             # fast beads and short steps: the contacts' forces (1e5) hardly turn them
    pos = ob.OracleSystem(_abi, cfg).read(ob.F_POS).reshape(-1, 4).copy()
    at = np.stack(np.meshgrid(*[np.arange(c) for c in cells], indexing="ij"), -1).reshape(-1, 3)
    pos[:, :3] = at * a + [0.1, 0.1, 12.0]
    vel = np.zeros_like(pos)
    vel[:, :3] = 2e4 * np.random.default_rng(2).normal(size=(n, 3))
    inner = (at[:, 2] >= 5) & (at[:, 2] < 10)
    state = {"positions": pos.astype(np.float32).ravel(), "velocities": vel.astype(np.float32).ravel(),
             "frozen": (~inner).astype(np.uint32)}
    runs = []
    for full in ("0", "1"):
        monkeypatch.setenv("SOUP_FULL_ROWS", full)
        g = SoupSystem(cfg, state)
        assert g.verlet_lists()[0].max() > 1400
        seen = [g.forces_no_rebuild()]
        for _ in range(4):
            g.debug_phase(_abi.PHASE_KICK_DRIFT)
            g.debug_phase(_abi.PHASE_FORCE)
            seen.append(g.forces_no_rebuild())
        assert 0.0 < g.info()["max_drift"] < 0.5 * cfg.skin
        assert rel_rms(seen[-1], g.forces_brute_force()) < FORCE_TOL
        runs.append(seen)
        g.dispose()
    for pruned, whole in zip(*runs):
        assert np.array_equal(pruned, whole)


@pytest.mark.parametrize("budget", [None, "0"])
@pytest.mark.parametrize("between", ["steps", "charges", "off-head charges", "bonds"])
def test_a_window_differentiates_its_own_charges_and_bonds(budget, between, monkeypatch):
    """the reverse pass behind other calls gives the gradient of the window, with every frame kept and with replays.
    Rows in another order round differently: 1e-6 a step, and 12 steps let it grow less than tenfold."""
    import torch
    if budget is not None:
        monkeypatch.setenv("SOUP_DIFF_FRAME_BUDGET_MB", budget)
    cfg, start = oracle_bilayer_start(steps=20)
    n = cfg.n
    assert (start["bond_slots"] != _abi.NONE).sum() > 100 and (start["charges"] != 0).sum() > 100
    g = SoupSystem(cfg, start)
    dldx = torch.randn((13, n, 4), generator=torch.Generator().manual_seed(1)).cuda()
    dldx[..., 3] = 0
    torch.cuda.synchronize()
    grads = []
    for other_calls in (False, True):
        g.write_state(start)
        g.diff_forward(12, 4)
        if other_calls:
            if between == "steps":
                g.step(40)
                g.protonation_sweep()
            elif between == "charges":
                g.write_charges(np.where(start["charges"] != 0, 0.0, np.where(start["positions"][3::4] == cfg.charged_kind, -1.0, 0.0)).astype(np.float32))
            elif between == "off-head charges":
                g.write_charges(np.full(n, 0.25, np.float32))
            else:
                g.write_state({"bond_slots": np.full(3 * n, _abi.NONE, np.uint32)})
        dx0, dv0 = torch.zeros((n, 4), device="cuda"), torch.zeros((n, 4), device="cuda")
        torch.cuda.synchronize()
        theta = g.diff_backward(dldx.data_ptr(), dx0.data_ptr(), dv0.data_ptr())
        torch.cuda.synchronize()
        grads.append((theta, dx0.cpu().numpy(), dv0.cpu().numpy()))
        assert np.array_equal(g.charges(), start["charges"]) and np.array_equal(g.bond_slots(), start["bond_slots"])
    for a, b in zip(*grads):
        assert np.abs(a).max() > 0
        if a.ndim == 1:
            assert np.all(np.abs(a - b) <= 1e-4 * np.abs(a).max()), (a, b)
        else:
            assert rel_rms(b, a) < 1e-4
    g.dispose()


def test_a_sweep_reads_lists_that_serve():
    """beads that moved beyond half the skin: the sweep's decisions are the oracle's on the positions of the moment"""
    def fixed(c):
        c.protonation_rng = 77
    cfg, o, g = make_pair(charged_opts(start={"C": 300, "O": 500, "H": 300, "M": 20, "W": 0}, rebuild_on_drift=True, skin=0.6,
                                       electrostatics={"enabled": True, "pH": 4.0}), relax=20, tweak=fixed)
    while g.info()["max_drift"] < 6.0:        # kicks and drifts alone: no step looks at the drift
        g.debug_phase(_abi.PHASE_KICK_DRIFT)
    now = ob.OracleSystem(_abi, cfg, dict(positions=g.particles(), charges=g.charges(), bond_slots=g.bond_slots(),
                                          center_link=g.center_links()))
    rg, ro = g.protonation_sweep(), now.sweep()
    assert np.array_equal(g.charges(), now.read(ob.F_CHARGES))
    assert g.protonation_rng_state() == int(now.read(ob.F_PROT_RNG)[0])
    assert rg["accepted"] == ro.accepted
    assert rg["dEsMeanKT"] == pytest.approx(ro.d_es_mean_kt, rel=1e-9, abs=1e-12)
    assert rel_rms(g.forces_no_rebuild(), now.forces64()) < FORCE_TOL
    g.dispose()


def test_site_energies_at_half_a_box():
    """a box below twice the cutoff, as a live box can shrink to, with heads half a box and up to 4e-7 apart: FP32
    rounds the offset to a half and takes the image on the other side.  The mean energy is FP64's to its fixed point."""
    opts = cfgm.SoupOptions(box=[20] * 3, seed=1, kT=1.1, start={"C": 0, "O": 100, "H": 0, "M": 1, "W": 0},
                            electrostatics={"enabled": True, "pH": 5.0, "ionicStrengthMolar": 0.01})
    cfg = cfgm.resolve(opts, P)
    cfg.box[0] = cfg.box[1] = cfg.box[2] = 16.0
    cfg.protonation_rng = 5
    cfg.es_list_capacity = 128
    assert cfg.es_cutoff > 8.5
    rng = np.random.default_rng(1)
    pos = ob.OracleSystem(_abi, cfg).read(ob.F_POS).reshape(-1, 4).copy()
    heads = np.nonzero(pos[:, 3] == cfg.charged_kind)[0]
    pos[:, :3] = rng.random((cfg.n, 3)) * [0.0, 3.0, 3.0]
    pos[heads[:50], 0] = np.float32(8.3)
    near = np.float32(8.3) - np.float32(8.0)
    pos[heads[50:], 0] = near - np.float32(2.0 ** -25) * rng.integers(1, 13, 50)
    pos = pos.astype(np.float32)
    apart = pos[heads[:1], 0].astype(np.float64) - pos[heads[50:], 0].astype(np.float64)
    assert np.all(apart > 8.0) and np.all((pos[heads[0], 0] - pos[heads[50:], 0]) == np.float32(8.0))
    q = np.zeros(cfg.n, np.float32)
    q[heads[::2]] = -1.0
    state = {"positions": pos.ravel(), "charges": q}
    o, g = ob.OracleSystem(_abi, cfg, state), SoupSystem(cfg, state)
    for k in range(3):
        rg, ro = g.protonation_sweep(), o.sweep()
        assert np.array_equal(g.charges(), o.read(ob.F_CHARGES)), k
        assert rg["accepted"] == ro.accepted > 0, k
        assert rg["dEsMeanKT"] == pytest.approx(ro.d_es_mean_kt, rel=1e-10, abs=1e-11), k
    g.dispose()


@pytest.mark.parametrize("boxes", [0, 3, 200, 50000])
@pytest.mark.parametrize("cutoff", [1.3, 4.0])
def test_aggregates_of_unwrapped_coordinates(boxes, cutoff):
    """coordinates written up to `boxes` boxes away: the reference takes the image in FP64"""
    side = 15.3
    opts = cfgm.SoupOptions(box=[side] * 3, seed=7, kT=1.1, start={"C": 600, "O": 0, "H": 0, "M": 1, "W": 0})
    cfg = cfgm.resolve(opts, P)
    rng = np.random.default_rng(boxes)
    pos = ob.OracleSystem(_abi, cfg).read(ob.F_POS).reshape(-1, 4).astype(np.float64)
    pos[:, :3] = rng.random((cfg.n, 3)) * side + side * rng.integers(-boxes, boxes + 1, (cfg.n, 3))
    pos = pos.astype(np.float32).ravel()
    g = SoupSystem(cfg, {"positions": pos})
    members = np.arange(0, cfg.n, 2 if cutoff < 2 else 29, dtype=np.uint32)
    n_o, lab_o = ob.aggregates(_abi, pos, members, cfg.box, cutoff)
    for labels in (g.aggregate_labels, g.aggregate_labels_noalloc):
        n_g, lab_g = labels(members, cutoff)
        assert n_g == n_o and np.array_equal(lab_g, lab_o)
    assert 1 < n_o < len(members)
    g.dispose()


def test_analysis_of_coordinates_that_are_no_numbers():
    """beads at infinity or at no number at all are aggregates of their own and leave the others' labels; a closure
    with some among its members and its water comes back"""
    opts = cfgm.SoupOptions(box=[15] * 3, seed=7, kT=1.1, start={"C": 300, "O": 0, "H": 0, "M": 1, "W": 0})
    cfg = cfgm.resolve(opts, P)
    pos = ob.OracleSystem(_abi, cfg).read(ob.F_POS).reshape(-1, 4).copy()
    pos[:, :3] = np.random.default_rng(3).random((cfg.n, 3)) * 15.0
    lost = np.array([0, 7, 150, 299])
    pos[lost, [0, 1, 2, 0]] = np.array([np.nan, np.inf, -np.inf, np.nan], np.float32)
    pos = pos.astype(np.float32)
    g = SoupSystem(cfg, {"positions": pos.ravel()})
    members = np.arange(cfg.n, dtype=np.uint32)
    kept = np.setdiff1d(members, lost).astype(np.uint32)
    n_o, lab_o = ob.aggregates(_abi, pos.ravel(), kept, cfg.box, 1.3)
    for labels in (g.aggregate_labels, g.aggregate_labels_noalloc):
        n_g, lab_g = labels(members, 1.3)
        assert n_g == n_o + len(lost) and np.array_equal(lab_g[kept], lab_o) and np.array_equal(lab_g[lost], lost)
    r = g.closure(members[:150], members[150:], [7.5, 7.5, 7.5], 0.5, 1.0, 0.5)
    assert r["totalEmptyCells"] > 0
    g.dispose()


def test_head_lists_of_a_sparse_box_over_rebuilds():
    """a million head cells for 200 heads, rebuilt over and over, and again after the grids were made anew: the cells'
    counts start at zero every time"""
    opts = cfgm.SoupOptions(box=[170] * 3, seed=2, kT=1.1, start={"C": 0, "O": 200, "H": 0, "M": 1, "W": 99},
                            electrostatics={"enabled": True, "pH": 7.0, "ionicStrengthMolar": 1.0}, rebuild_on_drift=True, skin=0.5)
    cfg = cfgm.resolve(opts, P)
    assert (170.0 / (cfg.es_list_range / 2)) ** 3 > 1e6
    rng = np.random.default_rng(2)
    pos = ob.OracleSystem(_abi, cfg).read(ob.F_POS).reshape(-1, 4).copy()
    pos[:, :3] = np.mod(np.repeat(rng.random((75, 3)) * 170.0, 4, axis=0) + rng.normal(size=(300, 3)), 170.0)
    pos = pos.astype(np.float32).ravel()
    g = SoupSystem(cfg, {"positions": pos})
    for again in range(4):
        if again == 2:
            g.set_box([170.0] * 3)
        g.debug_phase(_abi.PHASE_REBUILD)
        o = ob.OracleSystem(_abi, cfg, {"positions": g.particles()})
        for a, b in zip(g.es_lists(), o.es_lists()):
            assert np.array_equal(a, b)
    assert g.es_lists()[0].max() >= 2
    g.dispose()


@pytest.mark.parametrize("maker", ["replicas", "confined"])
def test_lanes_per_bead_change_no_bit_of_batches_and_parcels(maker, monkeypatch):
    """warps that span two replicas (bead counts that leave a remainder by every group), a parcel behind its wall, and
    the pass over the heads alone behind a sweep"""
    sched = dict(rebuild_on_drift=True, skin=1.0, sweep_every=4, chunk_steps=4)
    if maker == "replicas":
        start = {"C": 611, "O": 103, "H": 500, "M": 21, "W": 0}
        opts = [charged_opts(**sched), charged_opts(start=start, seed=8, **sched), charged_opts(seed=9, **sched)]
    else:
        opts = [confined_opts(**sched)]
    cfgs = [cfgm.resolve(o, P) for o in opts]
    states = []
    for cfg in cfgs:
        o = ob.OracleSystem(_abi, cfg)
        o.relax(20, 0.1)
        states.append(oracle_state(o))
    runs = []
    for lanes in ("4", "8", "16", "0"):
        monkeypatch.setenv("SOUP_TPP", lanes)
        b = SoupBatch(cfgs, states)
        b.step(8)                             # two sweeps
        runs.append([a for r in b.replicas for a in (r.particles(), r.velocities(), r.charges(), r.forces_no_rebuild())])
        for r in b.replicas:
            assert rel_rms(r.forces_no_rebuild(), r.forces_brute_force()) < FORCE_TOL
        b.dispose()
    for other in runs[1:]:
        for x, y in zip(runs[0], other):
            assert np.array_equal(x, y)


@pytest.mark.parametrize("n", [8191, 8200])
def test_a_dilute_system_steps_the_same_with_any_lanes(n, monkeypatch):
    """rows of a few entries on either side of the line from which they take four lanes"""
    opts = cfgm.SoupOptions(box=[70] * 3, seed=5, kT=1.1, start={"C": 0, "O": 0, "H": 0, "M": 1, "W": n - 1})
    cfg = cfgm.resolve(opts, P)
    pos = ob.OracleSystem(_abi, cfg).read(ob.F_POS)
    runs = []
    for lanes in ("0", "16"):
        monkeypatch.setenv("SOUP_TPP", lanes)
        g = SoupSystem(cfg, {"positions": pos})
        g.step(10)
        runs.append((g.particles(), g.forces_no_rebuild()))
        g.dispose()
    assert all(np.array_equal(a, b) for a, b in zip(*runs))


def _sweeps_are_the_oracles(g, cfg, sweeps=2):
    cfg.protonation_rng = g.protonation_rng_state()
    o = ob.OracleSystem(_abi, cfg, {"positions": g.particles(), "charges": g.charges()})
    for k in range(sweeps):
        rg, ro = g.protonation_sweep(), o.sweep()
        assert np.array_equal(g.charges(), o.read(ob.F_CHARGES)), k
        assert g.protonation_rng_state() == int(o.read(ob.F_PROT_RNG)[0]), k
        assert rg["accepted"] == ro.accepted > 0, k


@pytest.mark.parametrize("sides", [(40.0, 16.0, 40.0), (16.0, 40.0, 17.0)])
@pytest.mark.parametrize("heads", [100, 300, 1100])
def test_sweeps_in_a_live_box(sides, heads):
    """boxes in which the walk takes 512 and 256 draws a block, one after the other, in arrays laid out for the first"""
    cfg = cfgm.resolve(cfgm.SoupOptions(box=[sides[0]] * 3, seed=heads, kT=1.1, start={"C": 0, "O": heads, "H": 0, "M": 1, "W": 400},
                                        electrostatics={"enabled": True, "pH": 4.5, "ionicStrengthMolar": 0.1}), P)
    share = [cfg.es_cutoff ** 3 * 4.18879 / s ** 3 for s in sides]
    assert (min(share) < 0.06 < max(share)) and cfg.es_cutoff < 0.45 * 16
    cfg.protonation_rng = 3
    cfg.es_list_capacity = heads
    pos = ob.OracleSystem(_abi, cfg).read(ob.F_POS).reshape(-1, 4).copy()
    pos[:, :3] = np.random.default_rng(heads).random((cfg.n, 3)) * 15.9
    g = SoupSystem(cfg, {"positions": pos.astype(np.float32).ravel()})
    for k, side in enumerate(sides):
        if k:
            g.set_box([side] * 3)
            cfg.box[0] = cfg.box[1] = cfg.box[2] = side
        _sweeps_are_the_oracles(g, cfg)
    g.dispose()


def test_the_memory_of_many_small_replicas():
    """the sweep's arrays follow the replicas' own heads: 255 replicas of 20 heads took 1.3 GB for pairs that cannot be"""
    import torch
    cfgs = []
    for r in range(255):
        cfg = cfgm.resolve(cfgm.SoupOptions(box=[15] * 3, seed=r, kT=1.1, start={"C": 0, "O": 20, "H": 0, "M": 1, "W": 43},
                                            electrostatics={"enabled": True, "pH": 7.0, "ionicStrengthMolar": 0.1}), P)
        cfgs.append(cfg)
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    b = SoupBatch(cfgs)
    held = before - torch.cuda.mem_get_info()[0]
    b.replicas[254].protonation_sweep()
    b.dispose()
    assert held < 300e6, held

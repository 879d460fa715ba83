"""The constant-pH walk's blocks of draws at their edges: one and two heads (every draw of a block on the same
sites), head counts around half a block's draws (a sweep that ends inside, at and just behind a block), both
block sizes (by the share of the box the cutoff fills), a replica that walks alone and one with a group of
CTAs, and heads with a charge other than the deprotonated one.  Charges, the chain's state and the counts
equal the CPU oracle's exactly."""
import numpy as np
import pytest

import oracle_binding as ob
from protocell_genesis_b200 import _abi, config as cfgm
from protocell_genesis_b200.soup import SoupSystem

pytestmark = pytest.mark.gpu

P = cfgm.load_params()
# heads, box side, ionic strength: the cutoff is min(1.52 / sqrt(I), 0.45 box)
WIDE, NARROW = (20.0, 0.01), (40.0, 0.1)     # 0.38 and 0.0073 of the box: 256 and 512 draws a block


@pytest.mark.parametrize("heads", [1, 2, 100, 127, 128, 129, 300])
@pytest.mark.parametrize("box,ionic", [WIDE, NARROW])
@pytest.mark.parametrize("odd", [False, True])
def test_sweeps_at_the_edges_of_the_blocks(heads, box, ionic, odd):
    opts = cfgm.SoupOptions(box=[box] * 3, seed=heads, kT=1.1, start={"C": 0, "O": heads, "H": 0, "M": 1, "W": 400},
                            electrostatics={"enabled": True, "pH": 5.0, "ionicStrengthMolar": ionic})
    cfg = cfgm.resolve(opts, P)
    cfg.protonation_rng = 77 + heads
    cfg.es_list_capacity = max(64, heads)
    o = ob.OracleSystem(_abi, cfg)
    pos = o.read(ob.F_POS)
    q = o.read(ob.F_CHARGES)
    if odd:                                   # a few heads hold another charge, which a flip takes to 0
        at = np.nonzero(pos[3::4] == 1)[0]
        q[at[::5]] = -0.5
        o.write(ob.F_CHARGES, q)
    g = SoupSystem(cfg, {"positions": pos, "charges": q})
    for k in range(3):
        rg, ro = g.protonation_sweep(), o.sweep()
        assert np.array_equal(g.charges(), o.read(ob.F_CHARGES)), k
        assert g.protonation_rng_state() == int(o.read(ob.F_PROT_RNG)[0]), k
        assert rg["accepted"] == ro.accepted and rg["deprotonated"] == ro.deprotonated, k
        assert rg["dEsMeanKT"] == pytest.approx(ro.d_es_mean_kt, rel=1e-9, abs=1e-12), k
    g.dispose()
    o.close()


def test_a_batch_walks_both_block_sizes():
    cfgs, states, oracles = [], [], []
    from protocell_genesis_b200.soup import SoupBatch
    for k, (box, ionic) in enumerate((WIDE, NARROW, WIDE)):
        opts = cfgm.SoupOptions(box=[box] * 3, seed=3 + k, kT=1.1, start={"C": 0, "O": 150 + 90 * k, "H": 0, "M": 1, "W": 300},
                                electrostatics={"enabled": True, "pH": 5.0, "ionicStrengthMolar": ionic},
                                rebuild_on_drift=True, skin=1.0, sweep_every=4, chunk_steps=4)
        cfg = cfgm.resolve(opts, P)
        cfg.es_list_capacity = 400
        o = ob.OracleSystem(_abi, cfg)
        o.relax(30, 0.1)
        cfgs.append(cfg)
        states.append({"positions": o.read(ob.F_POS), "velocities": o.read(ob.F_VEL), "charges": o.read(ob.F_CHARGES),
                       "bond_rng": o.read(ob.F_BOND_RNG), "thermo_rng": o.read(ob.F_THERMO_RNG)})
    b = SoupBatch(cfgs, states)
    b.step(8)                                 # two sweeps of every replica
    for cfg, st, rep in zip(cfgs, states, b.replicas):
        s = SoupSystem(cfg, st)
        s.step(8)
        assert np.array_equal(rep.charges(), s.charges())
        assert np.array_equal(rep.particles(), s.particles())
        assert rep.protonation_rng_state() == s.protonation_rng_state()
        s.dispose()
    b.dispose()

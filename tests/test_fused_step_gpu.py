"""The fused kMC step at the edges of its shared-memory window, against single
replicas (the per-phase kernels), and the electrode sources' order against the
oracle on lattices one and two sites wide."""
import numpy as np
import pytest

import langmuir_b200 as L
from oracle.kmc_setup import independent_world, oracle_for

WINDOW = 1024  # carriers per species held in shared memory, at most


def params(**keys):
    base = dict(simulation_type="transistor", random_seed=11, seed_charges=1.0, coulomb_carriers=1,
                iterations_real=1000, iterations_print=10, grid_x=64, grid_y=64, grid_z=2,
                electron_percentage=0.15, hole_percentage=0.02, electrostatic_cutoff=10,
                voltage_right=1.0, e_source_l_rate=1.0, e_source_r_rate=1.0, e_drain_l_rate=0.01,
                e_drain_r_rate=0.01, h_drain_l_rate=0.5)
    base.update(keys)
    p = L.Params.default()
    for k, v in base.items():
        p.set(k, v)
    return p


def inner_sites(n, seed):
    """n distinct sites off the electrodes' faces of a 64x64x2 lattice."""
    s = np.arange(64 * 64 * 2)
    s = s[(s % 64 > 0) & (s % 64 < 63)]
    return np.random.default_rng(seed).choice(s, n, replace=False).astype(np.int32)


@pytest.mark.gpu
@pytest.mark.parametrize("start", [WINDOW - 10, WINDOW - 2, WINDOW + 40])
def test_window_edges_match_single_replicas(start):
    p, steps = params(), 30
    e, h = inner_sites(start, 3), inner_sites(40, 4)
    with L.KMCBatch([p], replica0=9, fused_max_charges=4096) as b:
        assert b.fused_count == 1
        b.replica(0).set_carriers(e, h)
        b.run(steps)
        (e1, h1), s1 = b.replica(0).carriers(), b.replica(0).stats()
    with L.KMC(p, replica=9) as k:
        k.set_carriers(e, h)
        k.run(steps)
        (e2, h2), s2 = k.carriers(), k.stats()
    assert len(e2) > WINDOW - 2  # past the window by the end
    np.testing.assert_array_equal(e1, e2)
    np.testing.assert_array_equal(h1, h2)
    assert s1["counters"] == s2["counters"]


@pytest.mark.gpu
def test_a_small_batch_leaves_a_large_one_its_window():
    big, small = params(), params(electron_percentage=0.005, hole_percentage=0.005)
    e, h = inner_sites(900, 3), inner_sites(40, 4)
    out = []
    for between in (False, True):
        with L.KMCBatch([big], replica0=2, fused_max_charges=4096) as b:
            b.replica(0).set_carriers(e, h)
            b.run(3)
            if between:
                with L.KMCBatch([small]) as c:
                    c.run(3)
            b.run(3)
            out.append(b.replica(0).carriers())
    np.testing.assert_array_equal(out[0][0], out[1][0])
    np.testing.assert_array_equal(out[0][1], out[1][1])


@pytest.mark.gpu
@pytest.mark.parametrize("x", [1, 2])
def test_sources_on_narrow_lattices_match_oracle(oracle_mod, x):
    """Both electrodes' faces are one face when the lattice is one site wide."""
    p = params(grid_x=x, grid_y=5, grid_z=2, electron_percentage=0.8, hole_percentage=0.8,
               seed_charges=0.0, h_source_l_rate=1.0, h_source_r_rate=1.0)
    with L.KMC(p, replica=4) as k:
        st = k.stats()
        e0, h0 = k.carriers()
        orc = oracle_for(oracle_mod, p, independent_world(p, 4), e0, h0, st["max_electrons"],
                         st["max_holes"], replica=4)
        for _ in range(40):
            orc.step()
        k.run(40)
        e, h = k.carriers()
        e_o, h_o = orc.carriers()
        np.testing.assert_array_equal(e, e_o)
        np.testing.assert_array_equal(h, h_o)
        np.testing.assert_array_equal(np.array(k.stats()["counters"], np.uint64), orc.counters)


@pytest.mark.gpu
@pytest.mark.parametrize("cap,keys", [
    (1, dict()), (511, dict()), (512, dict()), (513, dict()),  # 512^2 pairs is the line
    (295, dict(image_charges=3)), (296, dict(image_charges=3)),
    (200, dict(defects_charge=1, defect_percentage=0.02))])
def test_small_single_replicas_match_oracle(oracle_mod, cap, keys):
    """Both sides of the line between the one-block step and the separate kernels."""
    V = 64 * 64 * 2
    p = params(hole_percentage=(cap + 0.5) / V, electron_percentage=0.0, e_source_l_rate=0.0,
               e_source_r_rate=0.0, e_drain_l_rate=0.0, e_drain_r_rate=0.0, h_source_r_rate=0.7,
               h_drain_l_rate=0.9, **keys)
    with L.KMC(p, replica=6) as k:
        st = k.stats()
        assert st["max_holes"] == cap
        e0, h0 = k.carriers()
        orc = oracle_for(oracle_mod, p, independent_world(p, 6), e0, h0, st["max_electrons"],
                         st["max_holes"], replica=6)
        for n in (1, 7):  # a run after a run goes on where the first one ended
            for _ in range(n):
                orc.step()
            k.run(n)
            e, h = k.carriers()
            e_o, h_o = orc.carriers()
            np.testing.assert_array_equal(e, e_o)
            np.testing.assert_array_equal(h, h_o)
            np.testing.assert_array_equal(np.array(k.stats()["counters"], np.uint64), orc.counters)


@pytest.mark.gpu
@pytest.mark.parametrize("coulomb", [0, 1])
def test_rejected_source_tries_match_oracle(oracle_mod, coulomb):
    """Metropolis sources on faces that are nearly always full: tries that find
    their site taken follow one another without a pair sum between them."""
    p = params(grid_x=4, grid_y=3, grid_z=2, electron_percentage=0.6, hole_percentage=0.6,
               seed_charges=1.0, h_source_l_rate=1.0, h_source_r_rate=1.0, source_metropolis=1,
               source_coulomb=coulomb)
    with L.KMC(p, replica=5) as k:
        st = k.stats()
        e0, h0 = k.carriers()
        orc = oracle_for(oracle_mod, p, independent_world(p, 5), e0, h0, st["max_electrons"],
                         st["max_holes"], replica=5)
        for _ in range(200):
            orc.step()
        k.run(200)
        for got, want in zip(k.carriers(), orc.carriers()):
            np.testing.assert_array_equal(got, want)
        np.testing.assert_array_equal(np.array(k.stats()["counters"], np.uint64), orc.counters)

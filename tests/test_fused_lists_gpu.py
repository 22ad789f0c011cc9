"""The fused step past the list lengths where it claims sites and maps holes in global
arrays, and the forms of a batch without Coulomb sums, against the separate kernels."""
import numpy as np
import pytest

import langmuir_b200 as L

pytestmark = pytest.mark.gpu

LIST_MOST = 128  # kListMost


def _transistor(holes, X, Y, **kw):
    keys = dict(grid_x=X, grid_y=Y, grid_z=1, electron_percentage=0.0,
                hole_percentage=(holes + 0.5) / (X * Y), seed_charges=1.0, electrostatic_cutoff=10,
                voltage_right=1.0, e_source_l_rate=0.0, h_source_r_rate=0.9, h_drain_l_rate=0.9,
                random_seed=11)
    keys.update(kw)
    return L.Params.default(**keys)


def _solar(share, X, Y, **kw):
    keys = dict(simulation_type="solarcell", grid_x=X, grid_y=Y, grid_z=1,
                electron_percentage=share, hole_percentage=share, seed_charges=0.9,
                electrostatic_cutoff=10, voltage_right=0.5, generation_rate=0.5,
                source_scale_area=0.0, recombination_rate=0.02, recombination_range=1,
                random_seed=11)
    keys.update(kw)
    return L.Params.default(**keys)


def _same(params, steps, fused_max):
    with L.KMCBatch(params, device=0, fused_max_charges=fused_max) as a, \
            L.KMCBatch(params, device=0, fused_max_charges=0) as b:
        for n in (1, steps - 1):
            a.run(n)
            b.run(n)
        assert a.fused_count == len(params) and b.fused_count == 0
        stayed = 0
        for i in range(len(params)):
            ra, rb = a.replica(i), b.replica(i)
            sa, sb = ra.stats(), rb.stats()
            sa.pop("guard_evaluations"), sb.pop("guard_evaluations")
            assert sa == sb
            for x, y in zip(ra.carriers(), rb.carriers()):
                assert np.array_equal(x, y)
            stayed += sa["proposals"] - sa["accepted"]
        assert stayed > 0  # proposals that did not move their carrier


@pytest.mark.parametrize("coulomb", [0, 1])
@pytest.mark.parametrize("holes", [LIST_MOST - 1, LIST_MOST, LIST_MOST + 1, 300, 700])
def test_contested_sites(holes, coulomb):
    # a third of the lattice is filled: many accepted moves share a site
    Y = max(16, 3 * holes // 20)
    _same([_transistor(holes, 20, Y, coulomb_carriers=coulomb)] * 3, 60, 4096)


@pytest.mark.parametrize("coulomb", [0, 1])
@pytest.mark.parametrize("X,Y", [(20, 16), (40, 40)])
@pytest.mark.parametrize("reach", [1, 2])
def test_recombination(X, Y, reach, coulomb):
    # with 40 x 40 the lists pass the length, with 20 x 16 they stay below it
    _same([_solar(0.25, X, Y, coulomb_carriers=coulomb, recombination_range=reach)] * 3, 60, 4096)


@pytest.mark.parametrize("holes,X,Y", [(100, 40, 40), (600, 60, 60), (1100, 60, 60)])
def test_forms_without_coulomb_sums(holes, X, Y):
    # 128 threads; 256 threads; more holes than the window of shared memory
    _same([_transistor(holes, X, Y, coulomb_carriers=0)] * 5, 40, 4096)

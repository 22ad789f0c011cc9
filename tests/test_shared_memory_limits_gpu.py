"""Tables that bring a kernel's static and dynamic shared memory to either side of
the 48 KB a block gets unasked: FP64 entries at cutoffs 74 to 79, FP32 ones at 105
to 111.  Each kind of table in a process of its own, small tables first, since a
limit once raised stays raised for the process.

Tolerance: an FP32 weight is rounded once and added in runs of 16, so a sum is
within 17 2^-24 of its terms' magnitudes; in FP64 (test_fp64_sums_gpu) within
2 (n + 4) 2^-53."""
import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DIMS = (61, 47, 5)
N_SRC = 3000  # too many for the one-kernel form

CHILD = """
import sys
import numpy as np
import langmuir_b200 as L
z = np.load(sys.argv[1])
keys = dict(fp64=dict(precision=L.PREC_FP64), table64=dict(path=2), table=dict(path=1))[sys.argv[2]]
out = {}
for c in map(int, sys.argv[3:]):
    with L.Coulomb(*map(int, z["dims"]), cutoff=c, **keys) as ctx:
        out[str(c)] = ctx.potentials(z["src"], z["q"], z["tgt"], L.POINT, 7)
        assert ctx.last_launch()["kernel_launches"] == 7
        if sys.argv[2] != "fp64":
            ctx.autotune(len(z["src"]), len(z["tgt"]), L.POINT, 7)
np.savez(sys.argv[1] + ".out.npz", **out)
"""


@pytest.mark.parametrize("table,cutoffs", [("fp64", (74, 75, 78, 79)), ("table64", (74, 75, 78, 79)),
                                           ("table", (105, 106, 110, 111))])
def test_tables_around_the_default_limit(oracle_mod, tmp_path, table, cutoffs):
    rng = np.random.default_rng(5)
    V = DIMS[0] * DIMS[1] * DIMS[2]
    src = rng.choice(V, N_SRC, replace=False).astype(np.int32)
    q = rng.choice([-2, -1, 1, 3], N_SRC).astype(np.int32)
    tgt = rng.integers(0, V, 501).astype(np.int32)
    f = str(tmp_path / "in.npz")
    np.savez(f, dims=DIMS, src=src, q=q, tgt=tgt)
    r = subprocess.run([sys.executable, "-c", CHILD, f, table, *map(str, cutoffs)],
                       capture_output=True, text=True, timeout=300,
                       cwd=os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
    assert r.returncode == 0, r.stderr[-800:]
    got = np.load(f + ".out.npz")
    rel = 17 * 2.0 ** -24 if table == "table" else 2 * (N_SRC + 4) * 2.0 ** -53
    for c in cutoffs:
        orc = oracle_mod.Oracle(*DIMS, cutoff=c)
        want = orc.potentials(src, q, tgt, terms=7)
        direct = orc.potentials(src, np.abs(q), tgt, terms=1)
        norm = 2 * direct - orc.potentials(src, np.abs(q), tgt, terms=7)
        assert np.all(np.abs(got[str(c)] - want) <= rel * norm)


def gaussian_params(L, cutoff, sigma):
    return L.Params.default(grid_x=64, grid_y=64, grid_z=8, electron_percentage=0.03,
                            hole_percentage=0.03, seed_charges=1.0, coulomb_carriers=1,
                            electrostatic_cutoff=cutoff, coulomb_gaussian_sigma=sigma,
                            voltage_right=1.0, h_source_r_rate=0.9, h_drain_l_rate=0.9,
                            random_seed=3)


@pytest.mark.parametrize("first,then", [((50, 1.0), (20, 1.0)), ((30, 3.0), (30, 1.0))])
def test_a_gaussian_replica_leaves_an_older_one_its_tables(oracle_mod, first, then):
    """The older replica runs last, and steps as the oracle does."""
    import langmuir_b200 as L
    from oracle.kmc_setup import independent_world, oracle_for
    p = gaussian_params(L, *first)
    with L.KMC(p, replica=2) as a, L.KMC(gaussian_params(L, *then)) as b:
        b.run(2)
        st = a.stats()
        e0, h0 = a.carriers()
        orc = oracle_for(oracle_mod, p, independent_world(p, 2), e0, h0, st["max_electrons"],
                         st["max_holes"], replica=2)
        a.run(3)
        for _ in range(3):
            orc.step()
        for got, want in zip(a.carriers(), orc.carriers()):
            np.testing.assert_array_equal(got, want)


def test_a_gaussian_batch_leaves_an_older_one_its_tables():
    import langmuir_b200 as L
    out = []
    for between in (False, True):
        with L.KMCBatch([gaussian_params(L, 60, 8.0)], fused_max_charges=1) as a:
            if between:
                with L.KMCBatch([gaussian_params(L, 20, 1.0)], fused_max_charges=1) as b:
                    b.run(2)
            a.run(3)
            out.append(a.replica(0).carriers())
    for x, y in zip(*out):
        np.testing.assert_array_equal(x, y)

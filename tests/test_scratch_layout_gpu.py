"""The scratch of the chained kernels is cut anew for every call: calls of any sizes, paths
and variants on one context give what each gives on a context of its own, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DIMS = (50, 44, 12)
V = 50 * 44 * 12


@pytest.fixture(scope="module")
def lgm():
    import langmuir_b200
    return langmuir_b200


def draw(n, t, seed):
    rng = np.random.default_rng(seed)
    return (rng.choice(V, n, replace=False).astype(np.int32),
            rng.choice([-2, -1, 1, 3], n).astype(np.int32), rng.integers(0, V, t).astype(np.int32))


@pytest.mark.parametrize("keys", [dict(), dict(path=1), dict(path=2), dict(precision=1)])
def test_calls_of_all_sizes_share_a_context(lgm, keys):
    """Both block forms (2 MB is the line), growing and shrinking."""
    calls = [(2100, 300, 1), (2500, 40000, 7), (2100, 300, 1), (9000, 2000, 3), (64, 10, 7),
             (2048, 60000, 1), (2100, 5000, 5)]
    with lgm.Coulomb(*DIMS, cutoff=20, **keys) as ctx:
        for i, (n, t, terms) in enumerate(calls):
            src, q, tgt = draw(n, t, i)
            got = ctx.potentials(src, q, tgt, terms=terms)
            with lgm.Coulomb(*DIMS, cutoff=20, **keys) as own:
                np.testing.assert_array_equal(got, own.potentials(src, q, tgt, terms=terms))


def test_variants_and_tuning_share_a_context(lgm):
    src, q, tgt = draw(3000, 4000, 1)
    more = draw(7000, 9000, 2)
    with lgm.Coulomb(*DIMS, cutoff=20) as ctx:
        n = len(ctx.variants())
        for v in (0, 14, 32, n - 1):
            ctx.set_variant(v)
            got = ctx.potentials(src, q, tgt, terms=7)
            big = ctx.potentials(*more)
            with lgm.Coulomb(*DIMS, cutoff=20) as own:
                own.set_variant(v)
                np.testing.assert_array_equal(big, own.potentials(*more))
                np.testing.assert_array_equal(got, own.potentials(src, q, tgt, terms=7))
            np.testing.assert_array_equal(ctx.potentials(src, q, tgt, terms=7), got)
        ctx.set_variant(-1)
        ctx.autotune(3000, 4000, terms=7)
        tuned = ctx.potentials(src, q, tgt, terms=7)
        ctx.set_counting(True)
        np.testing.assert_array_equal(ctx.potentials(src, q, tgt, terms=7), tuned)

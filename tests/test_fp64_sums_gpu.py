"""FP64 precision on both sides of its table limit (cutoff 159 is the last with
tables), from the one-kernel form and the chained kernels, against the oracle
and against the kernel that computes every term (which counting calls take).

Tolerance: a sum of n FP64 terms, each rounded twice (square root, quotient; the
error function adds one more) and added in any order, is within (n + 4) 2^-53 of
the sum of the terms' magnitudes; the reference has the same error."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def lgm():
    import langmuir_b200
    return langmuir_b200


def draw(X, Y, Z, n, t, seed):
    rng = np.random.default_rng(seed)
    V = X * Y * Z
    src = rng.choice(V, n, replace=False).astype(np.int32)
    q = rng.choice([-2, -1, 1, 3], n).astype(np.int32)
    tgt = np.concatenate([src[:t // 2], rng.integers(0, V, t - t // 2 - 1), [V + 2]]).astype(np.int32)
    return src, q, tgt


@pytest.mark.parametrize("n,t", [(1, 1), (17, 33), (700, 301), (2049, 65)])
@pytest.mark.parametrize("cutoff,sigma,terms", [(9, 0.0, 7), (50, 0.0, 1), (40, 1.3, 1),
                                                (159, 0.0, 3), (160, 0.0, 3)])
def test_fp64_sums(lgm, oracle_mod, n, t, cutoff, sigma, terms):
    X, Y, Z = 61, 47, 5
    src, q, tgt = draw(X, Y, Z, n, t, n + cutoff)
    kind = lgm.GAUSS if sigma else lgm.POINT
    orc = oracle_mod.Oracle(X, Y, Z, cutoff=cutoff, sigma=sigma)
    want = orc.potentials(src, q, tgt, gauss=bool(sigma), terms=terms)
    norm = sum(np.abs(orc.potentials(src, np.abs(q), tgt, gauss=bool(sigma), terms=1 | k) -
                      (orc.potentials(src, np.abs(q), tgt, gauss=bool(sigma), terms=1) if k else 0))
               for k in (0, 2, 4) if k == 0 or terms & k)
    with lgm.Coulomb(X, Y, Z, cutoff=cutoff, sigma=sigma, precision=lgm.PREC_FP64) as ctx:
        got = ctx.potentials(src, q, tgt, kind, terms)
        info = ctx.last_launch()
        ctx.set_counting(True)
        direct = ctx.potentials(src, q, tgt, kind, terms)
        assert ctx.last_launch()["kernel_launches"] == 5
    assert info["variant"] == -1
    assert info["kernel_launches"] == (5 if cutoff > 159 else 7 if n > 2048 or cutoff == 159 else 1)
    tol = 2 * (n + 4) * 2.0 ** -53 * norm
    assert np.all(np.abs(got - direct) <= tol)
    assert np.all(np.abs(got - want) <= tol + 1e-300)


def test_a_small_cutoff_leaves_a_large_one_its_tables(lgm):
    """Shared-memory limits are the functions', shared by every context."""
    src, q, tgt = draw(61, 47, 5, 2049, 65, 8)
    with lgm.Coulomb(61, 47, 5, cutoff=150, precision=lgm.PREC_FP64) as a:
        one = a.potentials(src, q, tgt)
        with lgm.Coulomb(61, 47, 5, cutoff=90, precision=lgm.PREC_FP64) as b:
            b.potentials(src, q, tgt)
        np.testing.assert_array_equal(a.potentials(src, q, tgt), one)

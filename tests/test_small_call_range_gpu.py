"""Which calls of few sources take the one-kernel form, on both sides of its lines, and
that both forms add the same FP32 runs there (their FP64 order differs: 1e-13 of the
terms' magnitudes, as in test_mma_sums_gpu)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def lgm():
    import langmuir_b200
    return langmuir_b200


@pytest.mark.parametrize("n,t,path,one", [
    (512, 70000, 0, True), (513, 70000, 0, False), (513, 65000, 0, True), (512, 70000, 1, True),
    (512, 70000, 2, False), (512, 65536, 2, True), (1024, 32768, 0, True), (1024, 32769, 0, False),
    (1025, 4737, 0, False), (1025, 4736, 0, True), (2048, 4736, 0, True), (2048, 4737, 0, False)])
def test_both_sides_of_the_lines(lgm, n, t, path, one):
    dims = (40, 36, 9)
    V = 40 * 36 * 9
    rng = np.random.default_rng(n + t)
    src = rng.integers(0, V, n).astype(np.int32)
    q = rng.integers(-3, 4, n).astype(np.int32)
    tgt = rng.integers(0, V, t).astype(np.int32)
    with lgm.Coulomb(*dims, cutoff=15, path=path) as ctx:
        got = ctx.potentials(src, q, tgt)
        assert (ctx.last_launch()["kernel_launches"] == 1) == one
        ctx.set_variant(len(ctx.variants()) - 1)
        chain = ctx.potentials(src, q, tgt)
        norm = ctx.potentials(src, np.abs(q), tgt)
    assert np.all(np.abs(got - chain) <= 1e-13 * norm)


@pytest.mark.parametrize("n,path,one", [(1000, 0, True), (1024, 1, True), (1025, 0, False),
                                        (1000, 2, False)])
def test_every_site(lgm, n, path, one):
    dims = (64, 61, 30)
    V = 64 * 61 * 30
    rng = np.random.default_rng(n)
    src = rng.integers(0, V, n).astype(np.int32)
    q = rng.integers(-3, 4, n).astype(np.int32)
    with lgm.Coulomb(*dims, cutoff=15, path=path) as ctx:
        got = ctx.kernel1(src, q)
        assert (ctx.last_launch()["kernel_launches"] == 1) == one
        ctx.set_variant(len(ctx.variants()) - 1)
        chain = ctx.kernel1(src, q)
        norm = ctx.kernel1(src, np.abs(q))
    assert np.all(np.abs(got - chain) <= 1e-13 * norm)


def test_tuning_knows_the_one_kernel_form(lgm):
    """163 sources and targets: one kernel is far below half the chain's time, so tuning
    the size must not move it to the chain; nor every-site calls, which tuning does not
    time.  Larger sizes keep the variant found."""
    dims = (64, 61, 30)
    V = 64 * 61 * 30
    rng = np.random.default_rng(2)
    src = rng.choice(V, 3000, replace=False).astype(np.int32)
    q = rng.choice([-1, 1], 3000).astype(np.int32)
    with lgm.Coulomb(*dims, cutoff=15) as ctx:
        last = len(ctx.variants()) - 1
        before = ctx.potentials(src[:163], q[:163], src[:163])
        assert ctx.autotune(163, 163) == last
        np.testing.assert_array_equal(ctx.potentials(src[:163], q[:163], src[:163]), before)
        assert ctx.last_launch()["kernel_launches"] == 1
        ctx.autotune(1000, V)
        ctx.kernel1(src[:1000], q[:1000])
        assert ctx.last_launch()["kernel_launches"] == 1
        best = ctx.autotune(3000, 3000)
        ctx.potentials(src, q, src)
        assert ctx.last_launch()["variant"] == best
        # a tuned context keeps the settings it had
        ctx.set_variant(0)
        ctx.autotune(163, 163)
        ctx.potentials(src[:163], q[:163], src[:163])
        assert ctx.last_launch()["variant"] == 0

"""The one-kernel form's lines for calls on every site and for terms from FP64 tables: both
sides of each, and that both forms add the same terms there (FP32 runs alike, their FP64
order apart: 1e-13 of the terms' magnitudes, as in test_mma_sums_gpu)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SITES = {"below": (128, 126, 32), "at": (128, 128, 32)}  # 2^19 sites


def _charges(dims, n, t):
    V = dims[0] * dims[1] * dims[2]
    rng = np.random.default_rng(n + t)
    return (rng.integers(0, V, n).astype(np.int32), rng.integers(-3, 4, n).astype(np.int32),
            rng.integers(0, V, max(t, 1)).astype(np.int32))


@pytest.mark.parametrize("n,t,path,precision,one", [
    (512, 65536, 2, 0, True), (512, 65537, 2, 0, False), (513, 16352, 2, 0, True),
    (513, 16353, 2, 0, False), (1024, 8192, 2, 0, True), (1024, 8193, 2, 0, False),
    (1024, 8192, 0, 1, True), (1024, 8193, 0, 1, False), (1024, 8193, 1, 0, True)])
def test_given_targets(n, t, path, precision, one):
    import langmuir_b200 as lgm
    dims = (40, 36, 9)
    src, q, tgt = _charges(dims, n, t)
    with lgm.Coulomb(*dims, cutoff=15, path=path, precision=precision) as ctx:
        got = ctx.potentials(src, q, tgt)
        assert (ctx.last_launch()["kernel_launches"] == 1) == one
    with lgm.Coulomb(*dims, cutoff=15, path=path) as ctx:
        ctx.set_variant(len(ctx.variants()) - 1)
        chain, norm = ctx.potentials(src, q, tgt), ctx.potentials(src, np.abs(q), tgt)
    bound = 1e-13 if path or not precision else 1e-6  # FP64 precision against FP32 runs
    assert np.all(np.abs(got - chain) <= bound * norm)


@pytest.mark.parametrize("n,where,path,precision,one", [
    (1025, "at", 0, 0, True), (2048, "at", 0, 0, True), (2049, "at", 0, 0, False),
    (1025, "below", 0, 0, False), (1024, "below", 0, 0, True), (1025, "at", 1, 0, False),
    (400, "at", 2, 0, True), (401, "at", 2, 0, False), (400, "at", 0, 1, True),
    (401, "at", 0, 1, False)])
def test_every_site(n, where, path, precision, one):
    import langmuir_b200 as lgm
    dims = SITES[where]
    src, q, _ = _charges(dims, n, 0)
    with lgm.Coulomb(*dims, cutoff=12, path=path, precision=precision) as ctx:
        got = ctx.kernel1(src, q)
        assert (ctx.last_launch()["kernel_launches"] == 1) == one
    with lgm.Coulomb(*dims, cutoff=12, path=path) as ctx:
        ctx.set_variant(len(ctx.variants()) - 1)
        chain, norm = ctx.kernel1(src, q), ctx.kernel1(src, np.abs(q))
    bound = 1e-13 if path or not precision else 1e-6
    assert np.all(np.abs(got - chain) <= bound * norm)


def test_gaussian_sites_keep_the_chain():
    import langmuir_b200 as lgm
    dims = SITES["at"]
    src, q, _ = _charges(dims, 1025, 0)
    with lgm.Coulomb(*dims, cutoff=12, sigma=1.0) as ctx:
        ctx.kernel1(src, q, kind=lgm.GAUSS)
        assert ctx.last_launch()["kernel_launches"] > 1

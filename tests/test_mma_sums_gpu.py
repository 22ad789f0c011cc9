"""The pair sum with r^2 from the tensor cores (the default variant) against
the FP32 tile it replaces and against FP64 sums, at the edges of its exactness
and of its tiles."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL32, TOL64 = 1e-6, 1e-12


@pytest.fixture(scope="module")
def lgm():
    import langmuir_b200 as L
    return L


def fp32_tile(ctx):
    """The culled FP32 tile of the same FP32 run (16) without tensor cores."""
    vs = ctx.variants()
    return max(i for i, v in enumerate(vs[:-1]) if v["warp_specialised"] and v["run"] == 16)


def run_all(lgm, dims, cutoff, src, q, tgt, kind, terms, sigma=0.0, path=0):
    with lgm.Coulomb(*dims, cutoff=cutoff, sigma=sigma, path=path) as ctx:
        auto = ctx.potentials(src, q, tgt, kind, terms)
        info = ctx.last_launch()
        assert info["variant"] == len(ctx.variants()) - 1
        assert info["kernel_launches"] == (1 if len(src) <= 1300 else 7)
        ctx.set_variant(len(ctx.variants()) - 1)  # the chain, however few the sources
        got = ctx.potentials(src, q, tgt, kind, terms)
        assert ctx.last_launch()["kernel_launches"] == 7
        ctx.set_variant(fp32_tile(ctx))
        tile = ctx.potentials(src, q, tgt, kind, terms)
    with lgm.Coulomb(*dims, cutoff=cutoff, sigma=sigma, precision=lgm.PREC_FP64) as ctx:
        exact = ctx.potentials(src, q, tgt, kind, terms)
        norm = sum(abs(ctx.potentials(src, np.abs(q), tgt, kind, t)
                       - (0 if t == 1 else ctx.potentials(src, np.abs(q), tgt, kind, 1)))
                   for t in (1, 3, 5) if (t & terms) == t)
    # the same FP32 runs; only the FP64 order of the item partials differs
    assert np.all(np.abs(auto - got)[norm > 0] <= 1e-13 * norm[norm > 0])
    return got, tile, exact, norm


def check(got, tile, exact, norm, tol):
    # the same FP32 runs; only the FP64 order of the item partials differs
    assert np.all(np.abs(got - tile) <= 1e-13 * norm + 1e-300)
    assert np.all(np.abs(got - exact) <= tol * norm + 1e-300)


@pytest.mark.parametrize("dims,cutoff", [((418, 836, 2), 900), ((418, 3, 835), 900),
                                         ((2, 836, 3), 800), ((256, 256, 16), 50)])
def test_r2_exact_at_the_lattice_limit(lgm, dims, cutoff):
    """Largest accepted coordinates, images at both electrodes: every FP16 entry
    and FP32 partial sum of r^2 is at its largest; corners among the sites."""
    X, Y, Z = dims
    rng = np.random.default_rng(X + Y)
    V = X * Y * Z
    corners = [x + X * (y + Y * z) for x in (0, X - 1) for y in (0, Y - 1) for z in (0, Z - 1)]
    pool = np.setdiff1d(rng.choice(V, min(V, 3000), replace=False), corners)[:1200]
    src = np.concatenate([corners, pool[:len(pool) // 2]]).astype(np.int32)
    tgt = np.concatenate([src, pool]).astype(np.int32)
    q = rng.choice([-2, -1, 1, 3], len(src)).astype(np.int32)
    check(*run_all(lgm, dims, cutoff, src, q, tgt, lgm.POINT, 7), TOL32)


@pytest.mark.parametrize("n,t", [(1, 1), (15, 31), (16, 32), (17, 33), (127, 255), (128, 256),
                                 (129, 257), (400, 64), (1025, 1100)])
@pytest.mark.parametrize("kind,path", [(0, 0), (1, 0), (0, 1), (1, 1), (0, 2), (1, 2)])
def test_tile_and_chunk_edges(lgm, n, t, kind, path):
    """Numbers of sources and targets around a group, a chunk, a warp's and a
    tile's targets, for every path and kind; duplicate targets, drain ids."""
    dims = (40, 36, 9)
    V = 40 * 36 * 9
    rng = np.random.default_rng(n)
    src = rng.choice(V, n, replace=False).astype(np.int32)
    q = rng.choice([-1, 1], n).astype(np.int32)
    tgt = np.concatenate([rng.choice(V, t), src[:3], [V, V + 3]]).astype(np.int32)
    got, tile, exact, norm = run_all(lgm, dims, 20, src, q, tgt, kind, 3, sigma=1.2, path=path)
    check(got[:-2], tile[:-2], exact[:-2], norm[:-2], TOL64 if path == 2 else TOL32)
    np.testing.assert_allclose(got[-2:], tile[-2:], rtol=1e-12, atol=1e-15)


@pytest.mark.parametrize("n", [1, 63, 64, 65, 256, 257, 700, 2048, 2049])
@pytest.mark.parametrize("path", [0, 1, 2])
def test_one_kernel_call_at_its_edges(lgm, n, path):
    """Calls around the sizes of the one-kernel form (its sort's powers of two,
    its largest source count): host buffers, device buffers, every site, sources
    on one site, repeated calls, against the chain."""
    import torch
    dims = (30, 26, 7)
    V = 30 * 26 * 7
    rng = np.random.default_rng(n)
    src = rng.integers(0, V, n).astype(np.int32)  # several charges on a site: legal
    q = rng.integers(-3, 4, n).astype(np.int32)
    tgt = rng.integers(0, V, 77).astype(np.int32)
    with lgm.Coulomb(*dims, cutoff=17, path=path) as ctx:
        few = ctx.potentials(src, q, tgt, terms=7)
        assert (ctx.last_launch()["kernel_launches"] == 1) == (n <= 2048)
        for _ in range(3):
            np.testing.assert_array_equal(ctx.potentials(src, q, tgt, terms=7), few)
        site = ctx.kernel1(src, q)
        d = [torch.as_tensor(a).cuda() for a in (src, q, tgt)]
        out = torch.zeros(len(tgt), dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        ctx.potentials_async(d[0].data_ptr(), d[1].data_ptr(), n, d[2].data_ptr(), len(tgt),
                             out.data_ptr(), terms=7)
        ctx.sync()
        np.testing.assert_array_equal(out.cpu().numpy(), few)
        with pytest.raises(lgm.LgmError, match="source 0"):
            ctx.potentials(np.where(np.arange(n) == 0, V, src), q, tgt)
        with pytest.raises(lgm.LgmError, match="target 5"):
            ctx.potentials(src, q, np.where(np.arange(77) == 5, V + 35, tgt))
        ctx.set_variant(len(ctx.variants()) - 1)
        chain = ctx.potentials(src, q, tgt, terms=7)
        chain_site = ctx.kernel1(src, q)
        norm = ctx.potentials(src, np.abs(q), tgt) * 3 + 1e-300
        norm1 = ctx.kernel1(src, np.abs(q)) + 1e-300
    assert np.all(np.abs(few - chain) <= 1e-13 * norm)
    assert np.all(np.abs(site - chain_site) <= 1e-13 * norm1)

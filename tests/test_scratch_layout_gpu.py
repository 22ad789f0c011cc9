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


@pytest.mark.parametrize("n,warm,sizes", [(10000, 300000, (262000, 70000, 9000)),
                                          (4000, 262400, (262100, 131000)),
                                          (2622, 5244, (5000, 700))])
@pytest.mark.parametrize("precision", [0, 1])
def test_smaller_calls_are_captured_after_a_larger_one(lgm, n, warm, sizes, precision):
    """A captured call allocates nothing when a larger one has run, though fewer targets
    may be cut into more items (8192 segments of 32 targets are a line of that)."""
    import torch
    X, Y, Z = 128, 128, 24
    rng = np.random.default_rng(n)
    host = (rng.choice(X * Y * Z, n, replace=False).astype(np.int32),
            rng.choice([-1, 1], n).astype(np.int32),
            rng.integers(0, X * Y * Z, warm).astype(np.int32))
    src, q, tgt = (torch.as_tensor(a).cuda() for a in host)
    out = torch.zeros(warm, dtype=torch.float64, device="cuda")
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    with lgm.Coulomb(X, Y, Z, cutoff=20, precision=precision) as ctx:
        def call(t):
            ctx.potentials_async(src.data_ptr(), q.data_ptr(), n, tgt.data_ptr(), t,
                                 out.data_ptr(), stream=stream.cuda_stream)
        call(warm)
        ctx.sync(stream.cuda_stream)
        for t in sizes:
            g = torch.cuda.CUDAGraph()
            with torch.cuda.graph(g, stream=stream):
                call(t)
            out.zero_()
            torch.cuda.synchronize()
            g.replay()
            torch.cuda.synchronize()
            got = out[:t].cpu().numpy()
            np.testing.assert_array_equal(got, ctx.potentials(*host[:2], host[2][:t]))


@pytest.mark.parametrize("dims,cutoff,path,n,t,tile", [
    ((64, 64, 32), 50, 2, 2100, 32000, False), ((64, 64, 32), 50, 2, 2100, 65536, True),
    ((64, 64, 32), 50, 2, 2100, 66000, True), ((128, 128, 16), 20, 2, 2100, 65000, False),
    ((128, 128, 16), 20, 2, 2100, 66000, True), ((64, 64, 32), 100, 2, 2100, 7900, False),
    ((64, 64, 32), 100, 2, 2100, 8100, True), ((64, 64, 32), 100, 1, 2100, 8100, False),
    ((64, 64, 32), 150, 1, 2100, 7900, False), ((64, 64, 32), 150, 1, 2100, 8100, True),
    ((64, 64, 32), 40, 1, 2100, 199900, False), ((64, 64, 32), 40, 1, 2100, 200100, True),
    ((64, 64, 32), 39, 1, 2100, 200100, False), ((64, 64, 32), 150, 0, 2100, 250000, False),
    ((100, 90, 64), 64, 1, 2100, 200100, False), ((100, 90, 64), 65, 1, 2100, 200100, True)])
def test_which_kernel_sums_from_tables(lgm, dims, cutoff, path, n, t, tile):
    """Both sides of the lines between the two default kernels, which add the same FP32
    runs (or FP64 terms) in another order of FP64 sums; a smaller call on the same
    context may take the other kernel, under capture too."""
    import torch
    rng = np.random.default_rng(t)
    sites = dims[0] * dims[1] * dims[2]
    src = rng.choice(sites, n, replace=False).astype(np.int32)
    q = rng.choice([-2, -1, 1, 3], n).astype(np.int32)
    tgt = rng.integers(0, sites, t).astype(np.int32)
    with lgm.Coulomb(*dims, cutoff=cutoff, path=path) as ctx:
        last = len(ctx.variants()) - 1
        got = ctx.potentials(src, q, tgt)
        assert ctx.last_launch()["variant"] == (32 if tile else last)
        d = [torch.as_tensor(a).cuda() for a in (src, q, tgt)]
        out = torch.zeros(t, dtype=torch.float64, device="cuda")
        stream, g = torch.cuda.Stream(), torch.cuda.CUDAGraph()
        torch.cuda.synchronize()
        with torch.cuda.graph(g, stream=stream):
            ctx.potentials_async(d[0].data_ptr(), d[1].data_ptr(), n, d[2].data_ptr(), 5000,
                                 out.data_ptr(), stream=stream.cuda_stream)
        g.replay()
        torch.cuda.synchronize()
        few = out[:5000].cpu().numpy()
        ctx.set_variant(last if tile else 32)
        other = ctx.potentials(src, q, tgt)
        norm = ctx.potentials(src, np.abs(q), tgt)
    # FP64 sums of at most n terms or runs, rounded n times each
    assert np.all(np.abs(got - other) <= 2 * n * 2.0 ** -53 * norm)
    assert np.all(np.abs(few - got[:5000]) <= 2 * n * 2.0 ** -53 * norm[:5000])

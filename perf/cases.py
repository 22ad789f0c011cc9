"""Performance cases: what a user of langmuir_b200 has it do, through its public calls.

``listed()`` names twelve cases, ``draw(rng)`` gives more of the same ranges.  A case is a
dict of plain values; its ``what`` picks the path:

* ``sums``    ``Coulomb.kernel2`` / ``Coulomb.potentials`` on host arrays: the call an engine
              makes once per step through the OpenClHelper launch paths (host arrays in,
              potentials out), in every accumulation path;
* ``device``  ``Coulomb.potentials_async`` / ``kernel1_async`` on device arrays: a program that
              keeps its charges on the GPU, and the potential at every lattice site;
* ``kmc``     ``KMC.run``: one replica stepped on the GPU, its statistics and carriers read;
* ``batch``   ``KMCBatch.run`` over uneven replicas (parameter sweeps);
* ``labels``  ``KMCBatch.run`` over equal 2-D solar cells (the surrogate's training labels);
* ``train``   one mini-batch of the surrogate, forward and backward (``SurrogateFn``);
* ``screen``  ``Surrogate.predict`` over candidate morphologies.
"""
import math

import numpy as np
import torch

import langmuir_b200 as L
from langmuir_b200 import surrogate as S

PATHS = {"rsqrt": 0, "table": 1, "table64": 2}


# ---- the cases -----------------------------------------------------------------------------
def listed():
    return [
        # 163 holes on 128x128: the smallest replica an engine steps; latency decides
        dict(name="sums_2d_163", what="sums", X=128, Y=128, Z=1, cutoff=50, e=0, h=163, terms=1,
             sigma=0.0, path="rsqrt", precision=0, packed=True),
        # 21k charges on 256x256x16 with images at both electrodes: a full transistor
        dict(name="sums_3d_images_21k", what="sums", X=256, Y=256, Z=16, cutoff=50, e=10485,
             h=10485, terms=7, sigma=0.0, path="rsqrt", precision=0, packed=False),
        # Gaussian charges in a 128x128x64 solar cell, kernel-2 packing
        dict(name="sums_gauss_128x128x64", what="sums", X=128, Y=128, Z=64, cutoff=30, e=10485,
             h=10485, terms=1, sigma=1.0, path="rsqrt", precision=0, packed=True),
        # FP64 terms, the accuracy the engine's own comparison asks for, on a ragged lattice
        dict(name="sums_table64_ragged", what="sums", X=150, Y=131, Z=11, cutoff=50, e=1733,
             h=2011, terms=3, sigma=0.0, path="table64", precision=0, packed=False),
        # every term in FP64: the check of the last step's potentials
        dict(name="sums_fp64_check", what="sums", X=128, Y=128, Z=8, cutoff=50, e=1311, h=1311,
             terms=1, sigma=0.0, path="rsqrt", precision=1, packed=True),
        # the potential at every site of 256x256x16 (out.coulomb), resident on the device
        dict(name="map_256x256x16", what="device", X=256, Y=256, Z=16, cutoff=50, e=10485,
             h=10485, terms=1, sigma=0.0, path="rsqrt", precision=0, grid=True),
        # one small replica: 128x128 holes, launch-bound
        dict(name="kmc_2d_163", what="kmc", X=128, Y=128, Z=1, e=0.0, h=0.01, cutoff=50,
             sigma=0.0, images=0, solar=False, steps=200),
        # one large replica: 256x256x16, traps, disorder, images
        dict(name="kmc_3d_images_21k", what="kmc", X=256, Y=256, Z=16, e=0.01, h=0.01, cutoff=50,
             sigma=0.0, images=3, solar=False, steps=40),
        # a sweep: 512 uneven replicas advanced together
        dict(name="batch_512_uneven", what="batch", n=512, cutoff=50, steps=200),
        # label run of the surrogate: equal 128x128 solar cells after their burn-in
        dict(name="labels_1024", what="labels", n=1024, size=128, burn=2000, steps=3000),
        # one training mini-batch of the fit
        dict(name="train_64", what="train", B=64, H=128, W=128),
        # screening: an ensemble of four over new candidates
        dict(name="screen_4096", what="screen", n=4096, size=128, members=4),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _lattice(rng, most):
    """A lattice of at most `most` sites: thin films and blocks, odd sides among them."""
    while True:
        X, Y = _log(rng, 24, 256), _log(rng, 24, 256)
        Z = rng.choice([1, 1, 2, 4, 7, 8, 11, 16, 33, 64])
        if X * Y * Z <= most:
            return X, Y, Z


def draw(rng):
    what = rng.choice(["sums"] * 9 + ["device"] * 4 + ["kmc"] * 3 + ["batch", "labels"] +
                      ["train", "train", "screen"])
    if what in ("sums", "device"):
        fp64 = what == "sums" and rng.random() < 0.12
        grid = what == "device" and rng.random() < 0.5
        X, Y, Z = _lattice(rng, 1 << 17 if fp64 else 1 << 20)
        sigma = rng.choice([0.0, 0.0, 0.0, 1.0, 1.5]) if Z > 1 else 0.0
        n = max(4, min(int(X * Y * Z * rng.uniform(0.004, 0.03)), 3000 if fp64 else 20970))
        h = n if rng.random() < 0.3 else rng.randint(1, n)
        c = dict(what=what, X=X, Y=Y, Z=Z, cutoff=rng.choice([10, 20, 30, 50]), e=n - h, h=h,
                 terms=1 if grid or sigma else rng.choice([1, 1, 3, 7]), sigma=sigma,
                 path=rng.choice(["rsqrt", "rsqrt", "rsqrt", "table64", "table"]),
                 precision=int(fp64))
        if fp64:
            c["path"] = "rsqrt"
        c["grid" if what == "device" else "packed"] = grid if what == "device" else c["terms"] == 1
        return c
    if what == "kmc":
        X, Y, Z = _lattice(rng, 1 << 20)
        occ = rng.uniform(0.005, 0.02)
        holes_only = rng.random() < 0.3
        sigma = 1.0 if Z > 1 and rng.random() < 0.25 else 0.0
        solar = rng.random() < 0.3
        return dict(what="kmc", X=X, Y=Y, Z=Z, e=0.0 if holes_only and not solar else occ / 2,
                    h=occ if holes_only and not solar else occ / 2,
                    cutoff=rng.choice([20, 30, 50]), sigma=sigma,
                    images=0 if sigma or solar else rng.choice([0, 0, 1, 3]), solar=solar,
                    steps=rng.choice([20, 40, 60]))
    if what == "batch":
        return dict(what="batch", n=_log(rng, 16, 400), cutoff=rng.choice([30, 50]),
                    steps=rng.choice([100, 150, 200]))
    if what == "labels":
        return dict(what="labels", n=_log(rng, 32, 900), size=rng.choice([64, 96, 128]),
                    burn=rng.choice([500, 1000, 2000]), steps=rng.choice([1000, 2000, 3000]))
    H, W = rng.choice([(64, 128), (128, 128), (64, 256), (128, 256)])
    if what == "train":
        return dict(what="train", B=_log(rng, 3, 64 * 128 * 128 // (H * W)), H=H, W=W)
    return dict(what="screen", n=_log(rng, 50, 4000), size=128, members=rng.choice([1, 2, 4]))


# ---- inputs --------------------------------------------------------------------------------
def _charges(c, seed):
    """Seeded uniform placement and one nearest-neighbour proposal per carrier."""
    rng = np.random.default_rng(seed)
    X, Y, Z = c["X"], c["Y"], c["Z"]
    n = c["e"] + c["h"]
    sites = rng.choice(X * Y * Z, n, replace=False).astype(np.int64)
    q = np.concatenate([-np.ones(c["e"]), np.ones(c["h"])]).astype(np.int32)
    xyz = np.stack([sites % X, (sites // X) % Y, sites // (X * Y)], 1)
    dims = np.array([X, Y, Z])
    fut = xyz.copy()
    axis = rng.integers(0, 3 if Z > 1 else 2, n)
    fut[np.arange(n), axis] += rng.choice([-1, 1], n)
    off = (fut < 0) | (fut >= dims)
    fut[off] = 2 * xyz[off] - fut[off]  # reflect at the faces
    fs = fut[:, 0] + X * (fut[:, 1] + Y * fut[:, 2])
    return sites.astype(np.int32), q, np.concatenate([sites, fs]).astype(np.int32)


def _coulomb(c):
    return L.Coulomb(c["X"], c["Y"], c["Z"], cutoff=c["cutoff"], sigma=c["sigma"],
                     precision=c["precision"], path=PATHS[c["path"]])


def _kmc_params(c, seed):
    keys = dict(grid_x=c["X"], grid_y=c["Y"], grid_z=c["Z"], electron_percentage=c["e"],
                hole_percentage=c["h"], seed_charges=1.0, coulomb_carriers=1,
                electrostatic_cutoff=c["cutoff"], coulomb_gaussian_sigma=c["sigma"],
                random_seed=seed)
    if c["solar"]:
        keys.update(simulation_type="solarcell", seed_charges=0.8, voltage_right=0.5,
                    generation_rate=1e-3, source_scale_area=0.0, recombination_rate=1e-3,
                    recombination_range=1)
    else:
        keys.update(trap_percentage=0.02, trap_potential=0.2, site_disorder=0.05,
                    image_charges=c["images"], voltage_right=1.0, h_source_r_rate=0.9,
                    h_drain_l_rate=0.9)
        if c["e"] == 0:
            keys["e_source_l_rate"] = 0.0
    return L.Params.default(**keys)


def _batch_params(c, seed):
    """Side {32,64,128,256} x depth {1,2,4,8}, occupancy U(0.5%, 3%), voltage U(0.1, 2) V,
    traps U(0, 10%) at U(0.05, 0.3) eV; the sizes are the case's, the rest the seed's."""
    size, rng = np.random.default_rng(c["n"]), np.random.default_rng(seed)
    out = []
    for _ in range(c["n"]):
        xy, z = int(size.choice([32, 64, 128, 256])), int(size.choice([1, 2, 4, 8]))
        occ = float(size.uniform(0.005, 0.03))
        out.append(L.Params.default(
            grid_x=xy, grid_y=xy, grid_z=z, electron_percentage=occ / 2, hole_percentage=occ / 2,
            seed_charges=1.0, coulomb_carriers=1, electrostatic_cutoff=c["cutoff"],
            voltage_right=float(rng.uniform(0.1, 2.0)),
            trap_percentage=float(rng.uniform(0.0, 0.10)),
            trap_potential=float(rng.uniform(0.05, 0.3)), h_source_r_rate=0.9,
            h_drain_l_rate=0.9, random_seed=seed))
    return out


def prepare(case, seed):
    c = case
    if c["what"] in ("sums", "device"):
        src, q, both = _charges(c, seed)
        s = dict(c=c, ctx=_coulomb(c), n=len(src), kind=L.GAUSS if c["sigma"] > 0 else L.POINT)
        if c["what"] == "sums":
            s.update(src=src, q=q, both=both, q2=np.concatenate([q, q]),
                     out=np.empty(len(both), np.float64))
        else:
            dev = torch.device("cuda", 0)
            s["stream"] = torch.cuda.Stream()
            t = c["X"] * c["Y"] * c["Z"] if c["grid"] else len(both)
            s.update(src=torch.as_tensor(src, device=dev), q=torch.as_tensor(q, device=dev),
                     both=torch.as_tensor(both, device=dev), t=t,
                     out=torch.empty(t, dtype=torch.float64, device=dev))
            torch.cuda.synchronize()  # the inputs were made on another stream
        return s
    if c["what"] == "kmc":
        return dict(c=c, k=L.KMC(_kmc_params(c, seed), device=0, replica=seed % 1000))
    if c["what"] == "batch":
        b = L.KMCBatch(_batch_params(c, seed), device=0)
        return dict(c=c, b=b, reps=[b.replica(i) for i in range(c["n"])])
    if c["what"] == "labels":
        ph, _, _ = S.grf_morphologies(c["n"], size=c["size"], seed=seed)
        ph = ph.cpu().numpy()
        b = L.KMCBatch([S.solar_label_params(size=c["size"], seed=seed)] * c["n"], device=0)
        reps = [b.replica(i) for i in range(c["n"])]
        for r, p in zip(reps, ph):
            r.set_morphology(p.reshape(-1))
        b.run(c["burn"])
        return dict(c=c, b=b, reps=reps)
    if c["what"] == "train":
        g = torch.Generator(device="cuda").manual_seed(seed)
        ph, _, _ = S.grf_morphologies(c["B"], size=max(c["H"], c["W"]), seed=seed)
        return dict(c=c, x=S.phases_to_input(ph[:, :c["H"], :c["W"]].contiguous(), ramp=0.5),
                    y=torch.randn(c["B"], 2, generator=g, device="cuda"),
                    params=S.init_params(seed))
    ph, _, _ = S.grf_morphologies(c["n"], size=c["size"], seed=seed)
    return dict(c=c, ph=ph, model=S.Surrogate(members=c["members"], seed=seed, ramp=0.5))


# ---- one pass ------------------------------------------------------------------------------
def _counters(stats):
    return np.array([[s["step"], s["electrons"], s["holes"], s["proposals"], s["accepted"]] +
                     s["counters"] for s in stats], np.int64)


def _carriers(reps, stats):
    """Every replica's electron and hole sites, each list in room for its maximum."""
    room = [s[k] for s in stats for k in ("max_electrons", "max_holes")]
    out, at = np.full(sum(room), -1, np.int32), 0
    for a, n in zip((a for r in reps for a in r.carriers()), room):
        out[at:at + len(a)] = a
        at += n
    return out


def run(s):
    c = s["c"]
    if c["what"] == "sums":
        if c["packed"]:  # kernel 2: current sites then proposed ones, the first n the sources
            return s["ctx"].kernel2(s["both"], s["q2"], s["n"], kind=s["kind"], out=s["out"])
        return s["ctx"].potentials(s["src"], s["q"], s["both"], kind=s["kind"],
                                   terms=c["terms"], out=s["out"])
    if c["what"] == "device":
        st = s["stream"].cuda_stream
        if c["grid"]:
            s["ctx"].kernel1_async(s["src"].data_ptr(), s["q"].data_ptr(), s["n"],
                                   s["out"].data_ptr(), kind=s["kind"], stream=st)
        else:
            s["ctx"].potentials_async(s["src"].data_ptr(), s["q"].data_ptr(), s["n"],
                                      s["both"].data_ptr(), s["t"], s["out"].data_ptr(),
                                      kind=s["kind"], terms=c["terms"], stream=st)
        return s["out"]
    if c["what"] == "kmc":
        s["k"].run(c["steps"])
        stats = [s["k"].stats()]
        return {"counters": _counters(stats), "sites": _carriers([s["k"]], stats)}
    if c["what"] == "batch":
        s["b"].run(c["steps"])
        stats = [r.stats() for r in s["reps"]]
        return {"counters": _counters(stats), "sites": _carriers(s["reps"], stats)}
    if c["what"] == "labels":
        s["b"].run(c["steps"])
        return {"counters": _counters([r.stats() for r in s["reps"]])}
    if c["what"] == "train":
        pred = S.SurrogateFn.apply(s["x"], *s["params"])
        loss = ((pred - s["y"]) ** 2).mean()
        return {"pred": pred, "loss": loss, "grads": torch.autograd.grad(loss, s["params"])}
    mean, std = s["model"].predict(s["ph"])
    return {"mean": mean, "std": std}


# ---- the work of a pass --------------------------------------------------------------------
PAIR_FLOP = 11  # dx, dy, dz, r^2, 1/r, q/r + acc


def _inside(X, Y, Z, cutoff, terms=1):
    """Share of (target, source) pairs inside the cutoff, both placed uniformly, summed over
    the terms (an image pair lies x_t + x_s + 1 apart along x)."""
    def plain(n):
        d = np.arange(n)
        return d.astype(np.float64) ** 2, np.where(d > 0, 2.0, 1.0) * (n - d) / n ** 2
    (y2, py), (z2, pz) = plain(Y), plain(Z)
    yz, pyz = (y2[:, None] + z2).ravel(), (py[:, None] * pz).ravel()
    o = np.argsort(yz)
    yz, cum = yz[o], np.cumsum(pyz[o])

    def share(x2, px):
        k = np.searchsorted(yz, cutoff ** 2 - x2, side="left")
        return float(np.sum(px * np.where(k > 0, cum[np.maximum(k, 1) - 1], 0.0)))
    total = share(*plain(X))
    if terms & 6:
        d = np.arange(1, 2 * X)
        px = np.minimum(d, 2 * X - d) / X ** 2
        total += bin(terms & 6).count("1") * share(d.astype(np.float64) ** 2, px)
    return total


def _step_flops(n, X, Y, Z, cutoff, terms=1):
    return 2.0 * n * n * _inside(X, Y, Z, cutoff, terms) * PAIR_FLOP


def _net_flops(H, W):
    """Multiply-adds of the network on one image, twice: 9 and 288 taps per output value."""
    return 2.0 * 32 * H * W * (9 + 288 * (1 / 4 + 1 / 16 + 1 / 64))


def work(case):
    c = case
    if c["what"] in ("sums", "device"):
        n = c["e"] + c["h"]
        t = c["X"] * c["Y"] * c["Z"] if c.get("grid") else 2 * n
        f = _inside(c["X"], c["Y"], c["Z"], c["cutoff"], c["terms"])
        return {"bytes": 8.0 * n + (0 if c.get("grid") else 4.0 * t) + 8.0 * t,
                "flops": n * t * f * PAIR_FLOP}
    if c["what"] == "kmc":
        n = (c["e"] + c["h"]) * c["X"] * c["Y"] * c["Z"]
        terms = 1 | (2 if c["images"] & 1 else 0) | (4 if c["images"] & 2 else 0)
        return {"bytes": 16.0 * n * c["steps"],
                "flops": c["steps"] * _step_flops(n, c["X"], c["Y"], c["Z"], c["cutoff"], terms)}
    if c["what"] == "batch":  # the mean over the sides, depths and occupancies drawn
        f = n = 0.0
        for xy in (32, 64, 128, 256):
            for z in (1, 2, 4, 8):
                v = xy * xy * z
                n += 0.0175 * v / 16
                f += (0.0175 ** 2 + 0.025 ** 2 / 12) * v * v * 2 * PAIR_FLOP * \
                    _inside(xy, xy, z, c["cutoff"]) / 16
        return {"bytes": 16.0 * n * c["n"] * c["steps"], "flops": f * c["n"] * c["steps"]}
    if c["what"] == "labels":  # about 80 charges live in a 128x128 cell after the burn-in
        n = 80.0 * (c["size"] / 128) ** 2
        return {"bytes": 16.0 * n * c["n"] * c["steps"],
                "flops": c["n"] * c["steps"] * _step_flops(n, c["size"], c["size"], 1, 30)}
    if c["what"] == "train":  # forward, input gradients (none for layer 1), weight gradients
        px = c["B"] * c["H"] * c["W"]
        acts = 32 * 2.0 * px * (1 + 1 / 4 + 1 / 16 + 1 / 64)  # kept for the backward pass
        return {"bytes": 2.0 * px + 2 * acts,
                "flops": 3 * c["B"] * _net_flops(c["H"], c["W"]) - 2.0 * 32 * 9 * px}
    return {"bytes": c["n"] * c["size"] ** 2 + 16.0 * c["n"],
            "flops": c["n"] * c["members"] * _net_flops(c["size"], c["size"])}


# ---- the same in 64 bits -------------------------------------------------------------------
def _exact_sums(c, seed):
    src, q, both = _charges(c, seed)
    dev = torch.device("cuda", 0)
    X, Y, c2 = c["X"], c["Y"], float(c["cutoff"] ** 2)
    # the default electrostatic.prefactor: e / (4 pi eps_r eps_0 a), eps_r 3.5, 1 nm sites
    prefactor = 1.60217646e-19 / (4.0 * math.pi * 3.5 * 8.854187817e-12 * 1e-9)

    def xyz(s):
        s = torch.as_tensor(s, device=dev).long()
        return [v.double() for v in (s % X, (s // X) % Y, s // (X * Y))]
    tgt = np.arange(X * Y * c["Z"]) if c.get("grid") else both
    xs, ys, zs = xyz(src)
    xt, yt, zt = xyz(tgt)
    qd = torch.as_tensor(q, device=dev).double()
    out = torch.zeros(len(tgt), dtype=torch.float64, device=dev)
    step = max(1, (1 << 25) // len(src))
    for a in range(0, len(tgt), step):
        b = slice(a, a + step)
        dyz = (yt[b, None] - ys) ** 2 + (zt[b, None] - zs) ** 2
        for bit, sign in ((1, 1.0), (2, -1.0), (4, -1.0)):
            if not c["terms"] & bit:
                continue
            x = xt[b, None]
            dx = x - xs if bit == 1 else x + xs + 1 if bit == 2 else 2 * X - 1 - x - xs
            r2 = dx * dx + dyz
            on = (r2 > 0) & (r2 < c2)
            r = r2.sqrt()
            w = torch.erf(r / (math.sqrt(2.0) * c["sigma"])) / r if c["sigma"] > 0 else 1.0 / r
            out[b] += sign * (torch.where(on, w, torch.zeros_like(w)) @ qd)
    return prefactor * out


def _net64(x, params):
    """x [B,1,H,W] float64; params as SurrogateFn takes them, float64."""
    c1w, c1b, c2w, c2b, c3w, c3b, c4w, c4b, f1w, f1b, f2w, f2b = params

    def conv(x, w, b):  # w [32][(ky*3 + kx)*cin + c]
        k = w.reshape(32, 3, 3, x.shape[1]).permute(0, 3, 1, 2)
        return torch.relu(torch.nn.functional.conv2d(x, k, b, padding=1))
    pool = torch.nn.functional.avg_pool2d
    x = pool(conv(x, c1w, c1b), 2)
    x = pool(conv(x, c2w, c2b), 2)
    x = pool(conv(x, c3w, c3b), 2)
    g = conv(x, c4w, c4b).mean((2, 3))
    return torch.relu(g @ f1w.T + f1b) @ f2w.T + f2b


def exact(case, seed):
    c = case
    if c["what"] in ("sums", "device"):
        return _exact_sums(c, seed)
    if c["what"] in ("kmc", "batch", "labels"):
        return None
    if c["what"] == "train":
        s = prepare(c, seed)
        params = [p.detach().double().requires_grad_(True) for p in s["params"]]
        pred = _net64(s["x"].double().permute(0, 3, 1, 2), params)
        loss = ((pred - s["y"].double()) ** 2).mean()
        return {"pred": pred, "loss": loss, "grads": torch.autograd.grad(loss, params)}
    s = prepare(c, seed)
    x = s["ph"].double()[:, None] * 2 - 1
    x = x + s["model"].ramp * torch.linspace(-1, 1, c["size"], dtype=torch.float64, device=x.device)
    y = torch.stack([torch.cat([_net64(x[i:i + 128], [p.detach().double() for p in m])
                                for i in range(0, c["n"], 128)]) for m in s["model"].members])
    mean = torch.exp(y.mean(0))
    std = mean * y.std(0) if len(y) > 1 else torch.zeros_like(mean)
    return {"mean": mean, "std": std}

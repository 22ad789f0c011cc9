"""Replicas, batches and contexts made, run and destroyed while another thread captures a graph:
a replica's own first run captures its step, so threads with replicas of their own meet this."""
import threading

import numpy as np
import pytest
import torch

import langmuir_b200 as L

pytestmark = pytest.mark.gpu


def _params(side):
    return L.Params.default(grid_x=side, grid_y=side, grid_z=4, electron_percentage=0.02,
                            hole_percentage=0.02, seed_charges=1.0, coulomb_carriers=1,
                            electrostatic_cutoff=20, voltage_right=1.0, h_source_r_rate=0.9,
                            h_drain_l_rate=0.9, random_seed=3)


def _work():
    out = []
    with L.KMC(_params(64), device=0) as k:  # separate kernels: captures its step
        k.run(3)
        out += list(k.carriers())
    with L.KMCBatch([_params(64), _params(32)], device=0, fused_max_charges=0) as b:
        b.run(3)
        out += [a for i in range(2) for a in b.replica(i).carriers()]
    with L.Coulomb(64, 64, 4, cutoff=20) as c:
        out.append(c.kernel1(out[0], np.ones(len(out[0]), np.int32)))
    return out


def test_while_another_thread_captures():
    want = _work()
    x = torch.zeros(8, device="cuda")
    st, g, got = torch.cuda.Stream(), torch.cuda.CUDAGraph(), []

    def other():
        try:
            got.append(_work())
        except Exception as e:  # reported below: the capture has to end first
            got.append(e)

    torch.cuda.synchronize()
    with torch.cuda.graph(g, stream=st, capture_error_mode="thread_local"):
        x += 1
        t = threading.Thread(target=other)
        t.start()
        t.join()
        x += 1
    g.replay()
    torch.cuda.synchronize()
    assert not isinstance(got[0], Exception), got[0]
    for a, b in zip(got[0], want, strict=True):
        np.testing.assert_array_equal(a, b)
    assert torch.all(x == 2)

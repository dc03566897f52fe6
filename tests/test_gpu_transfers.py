"""Uploads and read-backs: pinned and pageable arrays in any mix, sizes around
the 8 MB staging chunk, other threads copying through the same chunks at the
same time, and the first grid sized for any placement of the block.  What is
read back before a step is what was uploaded, bit for bit (FP64)."""
import threading

import numpy as np
import pytest

import cases
from gpu_util import needs_gpu, run_oracle

pytestmark = [pytest.mark.gpu, needs_gpu]

CHUNK = 8 << 20


def _arrays(n, dim, seed):
    rng = np.random.default_rng(seed)
    a = {"x": rng.uniform(0.0, 0.3, (n, dim)), "v": rng.normal(size=(n, dim)),
         "F": np.eye(dim) + 0.01 * rng.normal(size=(n, dim, dim)), "B": rng.normal(size=(n, dim, dim)),
         "scalars": rng.uniform(size=(n, 6))}
    return a


def _pinned(a):
    import torch
    t = torch.empty(a.shape, dtype=torch.float64, pin_memory=True).numpy()
    t[...] = a
    return t


def _sim(dim):
    from matter_tests_b200.gpu import GpuSim
    sc = cases.apply(cases.block(dim, 2, n=4), plastic_model=cases.PM.DP, M=0.6)
    return GpuSim(sc.params)


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("n", [1, 255, CHUNK // 48 - 1, CHUNK // 48, CHUNK // 24 + 1, CHUNK // 8 + 3])
@pytest.mark.parametrize("pin", ["none", "all", "x", "FB"])
def test_round_trip(dim, n, pin):
    a = _arrays(n, dim, n % 1000)
    given = {k: _pinned(v) if pin == "all" or k in pin else v for k, v in a.items()}
    g = _sim(dim)
    for _ in range(2):  # into a new context and into its buffers again
        g.upload(*(given[k] for k in ("x", "v", "F", "B", "scalars")))
        got = g.particles()
        for k, v in a.items():
            np.testing.assert_array_equal(got[k], v, err_msg=k)
    g.close()


def test_threads_copy_through_the_same_chunks():
    errors = []

    def work(seed):
        try:
            a = _arrays(200_000 + seed, 3, seed)
            g = _sim(3)
            for _ in range(3):
                g.upload(*(a[k] for k in ("x", "v", "F", "B", "scalars")))
                got = g.particles()
                for k, v in a.items():
                    np.testing.assert_array_equal(got[k], v, err_msg=k)
            g.close()
        except Exception as e:  # reported by the main thread
            errors.append(e)

    ts = [threading.Thread(target=work, args=(s,)) for s in range(4)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not errors, errors


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("shift", [0.0, -3.7, 1234.5])
def test_first_grid_of_a_shifted_block(dim, shift):
    sc = cases.apply(cases.block(dim, 2, n=5), plastic_model=cases.PM.NoPlasticity)
    sc.x = sc.x + shift
    from matter_tests_b200.gpu import GpuSim
    g = GpuSim(sc.params)
    big = np.random.default_rng(0).uniform(-9.0, 9.0, size=(sc.Np, dim)) * 0.01
    g.upload(big)  # another extent first, in the same buffers
    g.upload(sc.x, sc.v, sc.F, sc.B, sc.scalars)
    g.set_scene_objects(sc)
    g.step(1)
    o = run_oracle(sc, 1)
    grid = g.grid()
    assert tuple(grid["dims"]) == tuple(o["g"]["dims"])
    assert np.array_equal(grid["x"], o["g"]["x"]) and np.array_equal(grid["y"], o["g"]["y"])
    g.close()

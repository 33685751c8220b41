"""The RWG basis of meshes whose vertices carry many edges: the same functions in the same order, in time that does not
grow with the square of a fan."""
import time

import numpy as np
import pytest

from oracle import bem_oracle as bo


def _fan(n, seed):
    """Two cones over one ring of n vertices, triangles in random order; the apexes are vertices 0 and 1."""
    a = 2 * np.pi * np.arange(n) / n
    v = np.concatenate([[[0, 0, 1.0], [0, 0, -1.0]], np.stack([np.cos(a), np.sin(a), 0 * a], 1)])
    i, j = 2 + np.arange(n), 2 + (np.arange(n) + 1) % n
    t = np.concatenate([np.stack([0 * i, i, j], 1), np.stack([0 * i + 1, j, i], 1)])
    return v, np.random.default_rng(seed).permutation(t).astype(np.int32)


@pytest.mark.parametrize("n", [3, 20, 31, 32, 33, 64, 65, 300])
def test_fans_match_the_oracle(n):
    import bem_b200 as bb
    v, t = _fan(n, n)
    r, o = bb.build_rwg(v, t), bo.build_rwg(v, t.astype(np.int64), "cpp")
    assert r["N"] == o["N"] == 3 * n
    for k in ("tri_p", "tri_m", "free_p", "free_m"):
        assert np.array_equal(r[k], o[k])
    assert np.allclose(r["length"], o["length"], rtol=1e-15, atol=0)


def test_a_large_fan_takes_no_square():
    import bem_b200 as bb
    t0 = time.perf_counter()
    N = bb.build_rwg(*_fan(200_000, 1))["N"]
    assert N == 600_000 and time.perf_counter() - t0 < 5.0  # 0.2 s; two minutes by insertion

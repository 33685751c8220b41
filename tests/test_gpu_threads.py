"""One context per host thread, on one device: calls whose kernels take different amounts of shared memory at a time."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_threads_with_other_sizes_do_not_disturb_each_other():
    import bem_b200 as bb
    import torch
    v, t = bb.icosphere(1.0, 2)
    RT, w = np.eye(3)[None], np.ones(1)
    failed = []

    def work(seed):
        ctx = bb.Context(0)
        try:
            rng = np.random.default_rng(seed)
            gs = [bb.Geometry(ctx, v, t, q) for q in (4, 13)]
            X = torch.view_as_complex(torch.randn((2, gs[0].n, 2), dtype=torch.float64, device="cuda",
                                                  generator=torch.Generator("cuda").manual_seed(7)))
            torch.cuda.synchronize()
            cases = [(g, k) for g in gs for k in (0.3, 25.0, 60.0)]  # 9 to 110 node pairs: 3 to 42 KB and more
            want = {}
            for i in range(400):
                c = int(rng.integers(len(cases)))
                g, k = cases[c]
                M = bb.mueller_from_solutions_dev(g, X, RT, w, complex(k), 1.0, ntheta=361)
                B = bb.rhs_planewave_dev(g, complex(k, 0.1), 1.0, RT).cpu().numpy()
                ref = want.setdefault(c, (M, B))
                assert np.array_equal(M, ref[0]) and np.array_equal(B, ref[1])
        except Exception as e:  # noqa: BLE001
            failed.append(repr(e))
        finally:
            ctx.close()

    threads = [threading.Thread(target=work, args=(s,)) for s in range(3)]
    for th in threads:
        th.start()
    for th in threads:
        th.join()
    assert not failed, failed

"""The cubic field from several host threads at once, each with a context of its own, on grids whose
blocks ask for different amounts of shared memory: every call succeeds and gives the bits of a call alone."""
import threading

import numpy as np
import pytest
import torch

from conftest import prepared_mesh

pytestmark = pytest.mark.gpu


def test_contexts_on_threads_of_their_own():
    from its_b200 import Context, Svo
    V, F, o, w = prepared_mesh("small")
    jobs = []
    # a point per cell of the octree (80 KB a block), and a few points within a cell (half of that)
    for R, width in ((20, 0.625), (3, 0.01)) * 3:
        svo = Svo(Context(0), V, F, 32, o, w)
        lam = torch.from_numpy(np.random.default_rng(R).standard_normal(svo.num_verts)).cuda()
        alone = torch.empty((R + 1) ** 3, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        svo.eval_grid_cubic(lam, o, width * w, R, out=alone)
        jobs.append((svo, lam, R, width, alone, torch.empty_like(alone)))
    failures = []

    def work(svo, lam, R, width, alone, out):
        try:
            for _ in range(4000):
                svo.eval_grid_cubic(lam, o, width * w, R, out=out)
        except Exception as e:
            failures.append("R = %d: %s" % (R, e))

    threads = [threading.Thread(target=work, args=j) for j in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failures
    for svo, lam, R, width, alone, out in jobs:
        assert torch.equal(out, alone)
        svo.close()

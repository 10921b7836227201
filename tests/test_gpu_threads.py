"""Two threads, each with a solver and a stream of its own, whose passes run
the same run-time-plan kernels with tiles of different sizes."""
import threading

import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu

# Z tiles of 52 and 105 KB
GRIDS = [(1029, 4, 1), (2058, 4, 1)]


def test_tiles_of_two_threads(eng, cuda):
    import torch
    work = []
    for i, g in enumerate(GRIDS):
        c = dict(grid=g, cell=(4e-9, 4e-9, 4e-9), msat=1.1e6, aexch=1.5e-11, alpha=0.5)
        m = torch.from_numpy(O.seeded_m(g, 60 + i, "random")).cuda()
        s = eng.Solver(eng.mmx_params(**c))
        h = torch.empty_like(m)
        torch.cuda.synchronize()
        s.field(m.data_ptr(), h.data_ptr())
        torch.cuda.synchronize()
        work.append((s, m, h, h.cpu().numpy(), torch.cuda.Stream()))
    errors = []
    start = threading.Barrier(len(work))

    def loop(s, m, h, st):
        start.wait()
        try:
            for _ in range(3000):
                s.field(m.data_ptr(), h.data_ptr(), st.cuda_stream)
        except Exception as e:
            errors.append(e)

    ts = [threading.Thread(target=loop, args=(s, m, h, st)) for s, m, h, _, st in work]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    torch.cuda.synchronize()
    assert not errors, errors
    for s, m, h, want, _ in work:
        assert np.array_equal(h.cpu().numpy(), want)
        s.close()

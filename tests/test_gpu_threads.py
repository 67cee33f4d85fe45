"""Charge solves of several host threads, each on its own stream, give the results
of one thread: the kernels whose blocks wait for one another take turns."""
import threading

import pytest
import torch

from _gpu_helpers import T, rel

pytestmark = pytest.mark.gpu


def _work(dev, k, reps=1):
    """Charges of one small and one middling system, by CG and by the dense solve."""
    from admp_b200 import synthetic
    from admp_b200.nblist import TorchNeighborList
    from admp_b200.qeq import QEqForceModule, matinv_optimize, pgrad_optimize
    out = []
    for nmol, box_len in ((20 + k, 13.0), (300, 21.0)):
        pos, box, chi, hard, eta, _ = synthetic.water_system(nmol, box_len, 3 + k)
        p, b, c, h, e = (T(x, dev) for x in (pos, box, chi, hard, eta))
        n = len(pos)
        C, v = torch.ones(1, n, dtype=torch.float64, device=dev), torch.zeros(1, dtype=torch.float64, device=dev)
        for _ in range(reps):
            nb = TorchNeighborList(6.0)
            pairs = nb(p, b)
            a = (p, b, c, h, e, pairs, nb.get_ds(), nb.get_buffer_scales(), C, v)
            m = QEqForceModule(6.0, 5e-4, eps=1e-12, max_iter=500)
            out = out[:1] if nmol == 300 else []
            out.append((pgrad_optimize(m, None, *a)[1].detach(), matinv_optimize(m, *a)[1].detach()))
    return out


def _threads(dev, n, reps):
    got, errors = [None] * n, []

    def body(k):
        try:
            with torch.cuda.stream(torch.cuda.Stream(dev)):
                got[k] = _work(dev, k, reps)
                torch.cuda.current_stream().synchronize()
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    ts = [threading.Thread(target=body, args=(k,)) for k in range(n)]
    [t.start() for t in ts]
    [t.join() for t in ts]
    assert not errors, errors
    return got


def test_threads_on_their_own_streams(cuda):
    got = _threads(cuda, 4, 5)
    for k, g in enumerate(got):
        for x, y in zip(g, _work(cuda, k)):
            # both solves within n eps (4e-10) over eigenvalues of 1 or more, of charges above 0.1
            assert rel(x[0], y[0]) < 1e-8 and rel(x[1], y[1]) < 1e-10


def test_first_calls_of_a_process_from_several_threads(cuda):
    """A fresh process whose first calls come from eight threads at once: each kernel's
    shared-memory limit is set before any of them launches it."""
    import os
    import subprocess
    import sys
    here = os.path.dirname(os.path.abspath(__file__))
    paths = [here, os.path.dirname(here), os.path.join(os.path.dirname(here), "torch-admp_b200")]
    code = (f"import sys; sys.path[:0] = {paths!r}\nimport torch\nfrom test_gpu_threads import _threads\n"
            "_threads(torch.device('cuda:0'), 8, 1)\nprint('all ran')\n")
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "all ran" in r.stdout, r.stderr[-2000:]

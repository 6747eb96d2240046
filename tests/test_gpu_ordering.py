"""What calls on plans wait for, and what they leave alone: work of the caller
that is pending on other streams, and captures of other threads."""
import threading

import numpy as np
import pytest
import torch

from openfpm_numerics_gb300 import _capi as C
from openfpm_numerics_gb300 import workloads as W
from openfpm_numerics_gb300.plan import DcpsePlan

pytestmark = pytest.mark.gpu

FAST64 = C.ASSEMBLE_FAST | C.STORE_OUT_F64


def test_a_capture_elsewhere_survives(cuda):
    """A thread builds, assembles and closes plans of several sizes while
    another thread's stream is captured in thread-local mode."""
    sets = [(side, *(torch.tensor(x, device="cuda") for x in W.lattice(side, 2, jitter=0.1, seed=side)))
            for side in (30, 31, 40, 30)]
    stream, out, errors = torch.cuda.Stream(), [], []
    x = torch.arange(1000, dtype=torch.float64, device="cuda")
    y = torch.zeros_like(x)

    def build():
        for side, p, h in sets:
            plan = DcpsePlan(2, [[(2, 0), (0, 2)]], stream=stream)
            plan.build_neighbors(p, 3.1 / (side - 1))
            plan.build_neighbors(p, 3.1 / (side - 1))
            plan.assemble(p, FAST64 | C.STORE_OUT_F32)
            out.append(plan.info()["nnz"])
            plan.close()

    def work():
        try:
            build()
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    build()
    alone, out = out, []
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=torch.cuda.Stream(), capture_error_mode="thread_local"):
        y.add_(x)
        t = threading.Thread(target=work)
        t.start()
        t.join()
        y.mul_(2.0)
    assert not errors, errors
    assert out == alone
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(y, 2.0 * x)

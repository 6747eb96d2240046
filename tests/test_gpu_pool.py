"""Plans share freed device memory between threads and streams: two threads
build, assemble, apply and destroy plans of changing sizes on streams of their
own, with the previous plan's work still in flight when its memory is released;
the results are those of plans used alone."""
import threading

import numpy as np
import pytest
import torch

from openfpm_numerics_gb300 import _capi as C
from openfpm_numerics_gb300 import workloads as W
from openfpm_numerics_gb300.plan import DcpsePlan

pytestmark = pytest.mark.gpu

FLAGS = C.ASSEMBLE_FAST | C.STORE_OUT_F64 | C.STORE_OUT_F32


def _one(side, stream, outs):
    pos, h = W.lattice(side, 2, jitter=0.1, seed=side)
    with torch.cuda.stream(stream):
        p = torch.tensor(pos, device="cuda")
        f = torch.tensor(np.sin(7 * pos[:, 0]) + pos[:, 1], device="cuda")
        plan = DcpsePlan(2, [[(2, 0), (0, 2)], [(1, 0)]], stream=stream)
        plan.build_neighbors(p, 3.1 * h)
        plan.assemble(p, FLAGS)
        outs.append((side, plan.apply(f, C.F32), plan.apply(f, C.F64)))
        plan.close()  # the applies may still run


def test_pool_between_threads_and_streams(cuda):
    sides = [20, 33, 21, 40, 22, 34] * 4
    ref = {}
    alone = []
    for s in sorted(set(sides)):
        _one(s, torch.cuda.Stream(), alone)
    torch.cuda.synchronize()
    for s, a, b in alone:
        ref[s] = (a.clone(), b.clone())
    got, errors = [[], []], []

    def work(i):
        try:
            stream = torch.cuda.Stream()
            for s in (sides if i else sides[::-1]):
                _one(s, stream, got[i])
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert not errors, errors
    for outs in got:
        assert len(outs) == len(sides)
        for s, a, b in outs:
            assert torch.equal(a, ref[s][0]) and torch.equal(b, ref[s][1]), s

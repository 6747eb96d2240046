"""What calls on plans wait for, and what they leave alone: work of the caller
that is pending on other streams, and captures of other threads."""
import threading

import numpy as np
import pytest
import torch

from openfpm_numerics_gb300 import _capi as C
from openfpm_numerics_gb300 import operators as O
from openfpm_numerics_gb300 import workloads as W
from openfpm_numerics_gb300.odeint import GrayScottRK4
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


# about 5 ms of a bounded spin kernel: work of the caller on another stream
SPIN = 10_000_000


def _pending(stream):
    with torch.cuda.stream(stream):
        torch.cuda._sleep(SPIN)
        e = torch.cuda.Event()
        e.record(stream)
    assert not e.query()
    return e


def test_calls_that_replace_arrays_wait_for_the_device(cuda):
    """A new list, a re-assembly, a change of numbering, loaded kernels and a
    closed plan: the caller's work on other streams (which may read the plan's
    arrays, or write the call's inputs) is done before anything is replaced."""
    other = torch.cuda.Stream()
    pos, h = W.lattice(30, 2, jitter=0.1, seed=81)
    p = torch.tensor(pos, device="cuda")
    plan = DcpsePlan(2, [[(2, 0), (0, 2)]], stream=torch.cuda.Stream())
    plan.build_neighbors(p, 3.1 * h)
    full = C.STORE_TERMS_F64 | C.STORE_OUT_F64 | C.STORE_OUT_F32
    plan.assemble(p, full)
    rp, cols = (x.clone() for x in plan.neighbors())
    K, eip = (x.clone() for x in plan.term_kernels(0))
    eps = plan.eps()[0].clone()
    torch.cuda.synchronize()
    calls = {
        "assemble": lambda: plan.assemble(p, full | C.ASSEMBLE_ASYNC),
        "set_reorder": lambda: plan.set_reorder(1),
        "set_term_kernels": lambda: plan.set_term_kernels(0, K, eps, eip),
        "set_neighbors": lambda: plan.set_neighbors(rp, cols),
        "build_neighbors": lambda: plan.build_neighbors(p, 3.1 * h),
        "set_support": lambda: plan.set_support(None),
        "close": plan.close,
    }
    for name, call in calls.items():
        e = _pending(other)
        call()
        assert e.query(), name


def test_weights_read_on_another_stream_survive_a_reassembly(cuda):
    pos, h = W.lattice(40, 2, jitter=0.1, seed=82)
    p = torch.tensor(pos, device="cuda")
    moved = p + 0.01 * h
    moved[::2] -= 0.02 * h
    plan = DcpsePlan(2, [[(2, 0), (0, 2)]])
    plan.build_neighbors(p, 3.1 * h)
    plan.assemble(p, FAST64 | C.STORE_OUT_F32)
    w64, w32 = plan.output_weights(0)
    ref = w64.clone(), w32.clone()
    torch.cuda.synchronize()
    reader = torch.cuda.Stream()
    with torch.cuda.stream(reader):
        torch.cuda._sleep(SPIN)
        got = w64.clone(), w32.clone()
    plan.assemble(moved, FAST64 | C.STORE_OUT_F32)
    torch.cuda.synchronize()
    assert torch.equal(got[0], ref[0]) and torch.equal(got[1], ref[1])
    assert not torch.equal(plan.output_weights(0)[0], ref[0])
    plan.close()


def test_operator_updates_on_a_side_stream(cuda):
    """Operator objects updated inside torch.cuda.stream(s), with work pending on
    s and free blocks of the right sizes left by an operator of the same size:
    the lists and results of the same updates on the default stream."""
    rng = np.random.default_rng(83)
    pos, h = W.lattice(40, 2, jitter=0.1, seed=83)
    rc = 3.9 * h  # (nine neighbours or more in the corners of the moved sets)
    steps = [torch.tensor(pos + rng.uniform(-0.1 * h, 0.1 * h, pos.shape), device="cuda") for _ in range(4)]
    dom = torch.tensor(W.lattice(38, 2, h=h, origin=0.7 * h)[0], device="cuda")
    f = torch.tensor(rng.standard_normal(pos.shape[0]), device="cuda")
    box = dict(box=((-0.1, -0.1), (1.1, 1.1)))

    def run(pending):
        out = []
        parts = O.ParticleSet(steps[0], **box)
        target = O.ParticleSet(dom, **box)
        vl, vl2 = parts.getVerlet(rc), O.createVerletTwoPhase(target, parts, rc)
        spare = O.Laplacian(parts, vl, 2, rc)
        op = O.Laplacian(parts, vl, 2, rc)
        gpu = O.Laplacian_gpu(parts, vl, 2, rc)
        pp = O.PPInterpolation(parts, target, vl2, 2, rc)
        spare.deallocate()
        for x in steps[1:]:
            pending()
            parts.setPos(x + 0.0)  # (written on the current stream, after the pending work)
            op.update(parts, parts.getVerlet(rc))
            gpu.update(parts)
            pp.update(O.createVerletTwoPhase(target, parts, rc))
            for o in (op, gpu, pp):
                torch.cuda.synchronize()
                out.append(o(f))
                torch.cuda.synchronize()
                out += [o.verletList.rowptr, o.verletList.cols, *(t.clone() for t in o.plan.neighbors())]
        torch.cuda.synchronize()
        return out

    ref = run(lambda: None)
    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        got = run(lambda: torch.cuda._sleep(SPIN))
    assert len(ref) == len(got)
    assert all(torch.equal(a, b) for a, b in zip(ref, got))


def test_adjoint_prepared_again_on_another_stream(cuda):
    """Adjoint stages pending on one stream keep their weights while the adjoint
    is prepared again, for other weights, on another."""
    n = 16
    pos = np.mod(W.lattice(n, 3, h=1.0 / n, jitter=0.1, seed=84)[0], 1.0)
    p = torch.tensor(pos, device="cuda")
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    plan = DcpsePlan(3, [[(2, 0, 0), (0, 2, 0), (0, 0, 2)]], box=((0.0,) * 3, (1.0,) * 3, (1,) * 3), stream=a)
    plan.build_neighbors(p, 2.8 / n)
    flags = C.ASSEMBLE_FAST | C.STORE_OUT_F32
    plan.assemble(p, flags)
    g = torch.Generator(device="cuda").manual_seed(84)
    u, v, ub, vb = (torch.rand(n ** 3, generator=g, device="cuda") for _ in range(4))
    gs = GrayScottRK4(plan, u, v, 2e-5, 1e-5, 0.04, 0.06, 1.0)
    gs.prepare_adjoint()
    stages = [(u, v)] * 4
    torch.cuda.synchronize()

    def reverse(spin):
        with torch.cuda.stream(a):
            yb, acc = (ub.clone(), vb.clone()), (torch.empty_like(u), torch.empty_like(v))
            torch.cuda._sleep(spin)
            gs._reverse_step_into(stages, yb, acc)
        return yb

    ref = reverse(0)
    torch.cuda.synchronize()
    got = reverse(SPIN)
    plan.set_stream(b)
    plan.assemble(torch.remainder(p * 1.0 + 0.01 / n * torch.sin(40 * p), 1.0), flags | C.ASSEMBLE_ASYNC)
    gs.prepare_adjoint()
    torch.cuda.synchronize()
    assert torch.equal(ref[0], got[0]) and torch.equal(ref[1], got[1])
    plan.close()


def test_position_vjp_beside_a_pending_assembly(cuda):
    """The position VJP needs nothing of an assembly: on another stream it may
    run before, during or after one that is pending, and changes none of it."""
    pos, h = W.lattice(20, 3, jitter=0.1, seed=85)
    p = torch.tensor(pos, device="cuda")
    rng = np.random.default_rng(85)
    f = torch.tensor(rng.standard_normal(pos.shape[0]), device="cuda")
    outs = W.grad_lap_outputs(3)
    g = torch.tensor(rng.standard_normal((len(outs), pos.shape[0])), device="cuda")
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    plan = DcpsePlan(3, outs, stream=a)
    plan.build_neighbors(p, 2.8 * h)
    plan.assemble(p, FAST64)
    w = [plan.output_weights(o)[0] for o in range(len(outs))]
    ref, grad = [x.clone() for x in w], plan.vjp_positions(p, f, g)
    torch.cuda.synchronize()
    for spin in (SPIN, 0):
        for x in w:
            x.zero_()
        torch.cuda.synchronize()
        with torch.cuda.stream(a):
            torch.cuda._sleep(spin)
        plan.set_stream(a)
        plan.assemble(p, FAST64 | C.ASSEMBLE_ASYNC)
        plan.set_stream(b)
        got = plan.vjp_positions(p, f, g)
        torch.cuda.synchronize()
        assert torch.equal(got, grad)
        assert all(torch.equal(x, r) for x, r in zip(w, ref))
    plan.close()


def test_plans_destroyed_inside_a_capture(cuda):
    """Plans that end while this thread captures, the last one too, leave the
    capture alone."""
    pos, h = W.lattice(20, 2, jitter=0.1, seed=87)
    p = torch.tensor(pos, device="cuda")
    plans = []
    for _ in range(2):
        plans.append(DcpsePlan(2, [[(1, 0)]], stream=torch.cuda.Stream()))
        plans[-1].build_neighbors(p, 3.1 * h)
        plans[-1].assemble(p, FAST64)
    x, y = torch.ones(100, device="cuda"), torch.zeros(100, device="cuda")
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        y.add_(x)
        for plan in plans:
            plan.close()
        y.mul_(2.0)
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(y, 2.0 * x)


def test_released_memory_can_be_given_back(cuda):
    keep = DcpsePlan(2, [[(1, 0)]])
    pos, h = W.lattice(48, 3, jitter=0.1, seed=86)
    p = torch.tensor(pos, device="cuda")
    plan = DcpsePlan(3, W.grad_lap_outputs(3))
    plan.build_neighbors(p, 2.8 * h)
    plan.assemble(p, FAST64)
    plan.close()
    torch.cuda.synchronize()
    held = torch.cuda.mem_get_info()[0]
    cuda.release_memory()
    assert torch.cuda.mem_get_info()[0] - held > 200 << 20  # (the weights alone take 250 MB)
    keep.close()

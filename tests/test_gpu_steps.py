"""Many steps in one persistent launch (``csrc/steps.cu``) against the step-by-step launches.

Both run the same equations from the same state; they differ in the order of
the float64 sums over rows, in the stopping test (formed from the sums of the
pass instead of a second reduction) and in r' taken from float32 pairs, each a
relative 1e-12 or less of what is rounded to float32 once.  So after a stretch
of steps the solutions agree to a few float32 ulp of their range per step:
steps * 2^-23 is the bound used, and the iteration counts are equal.
"""
import ctypes as C

import numpy as np
import pytest
import torch

from torchcor_b200 import meshgen

pytestmark = pytest.mark.gpu


def _sim(mesh, size, model, device, theta=0.5, dt=0.02, steps=160):
    from torchcor_b200.ionic import CourtemancheRamirezNattel, ModifiedMS2v, TenTusscherPanfilov
    from torchcor_b200.simulator import Monodomain
    if model == "ttp":
        im = TenTusscherPanfilov("ENDO", dt, device=device)
    elif model == "crn":
        im = CourtemancheRamirezNattel(dt, device=device)
    else:
        im = ModifiedMS2v(dt, device=device)
    sim = Monodomain(im, T=(steps + 0.5) * dt, dt=dt, device=device)
    sim.theta = theta
    if mesh == "cube":
        nodes, elems = meshgen.cube(size, 0.25)
        fib = meshgen.fibres_constant(len(elems))
    else:
        nodes, elems = meshgen.icosphere_fast(size, 25.0)
        fib = meshgen.fibres_random_tangent(nodes, elems, 3)
    sim.load_arrays(nodes / 1000.0, elems, np.ones(len(elems), dtype=np.int64), fib)
    sim.add_conductivity([1], il=0.5, it=0.2)
    sim.add_stimulus(None, 0.0, 1.0, 100, region=np.arange(max(1, len(nodes) // 9)))
    return sim


def _run(sim, tol, max_iter, guess, fused_step, chunks, frames=False):
    from torchcor_b200._lib import check, load, stream_ptr
    sim._sim = None
    sim.prepare(tol, tol, max_iter, linear_guess=guess, snapshot_interval=1 if frames else sim.T)
    sim.set_launch(fused_step=fused_step)
    for k in chunks:
        sim.run_steps(k)
    check(load().tcb_mono_check(C.byref(sim._sim["struct"]), stream_ptr()))
    assert (sim._sim["work"] is not None) == (fused_step == 0)
    d = sim._sim
    n = sim.n_nodes
    out = dict(x=d["x"][:, :n].clone(), state=sim.ionic_model.state[:, :n].clone(), at=d["at"].clone(), rt=d["rt"].clone(),
               iters=d["step_iters"].clone())
    if frames:
        out["frames"] = d["snaps"][: sim._frames_written() + 1].clone()
    return out


@pytest.mark.parametrize("mesh,size,model,tol,max_iter,guess,theta", [
    ("cube", 2, "ms", 1e-5, 100, True, 0.5),        # 27 nodes: one ragged slice, one block
    ("cube", 7, "ttp", 1e-5, 100, True, 0.5),       # 512 nodes: whole slices
    ("cube", 9, "crn", 1e-8, 100, False, 0.5),      # many passes a step
    ("cube", 11, "ms", 1e-8, 2, True, 0.5),         # stopped by max_iter
    ("cube", 11, "ms", 1e-5, 0, True, 0.5),         # no pass at all
    ("cube", 15, "crn", 1e-6, 100, True, 0.5),      # 4,096 nodes: a full cluster of 16 blocks, whole slices
    ("cube", 16, "ttp", 1e-6, 100, True, 0.5),      # 4,913 nodes: the smallest grid
    ("cube", 13, "ttp", 1e-6, 100, True, 0.25),     # A is not M Cm + K'
    ("ico", 3, "crn", 1e-6, 100, True, 0.5),        # rows of 6 and 7 entries
    ("ico", 6, "ms", 1e-6, 100, True, 0.5),         # 32-bit columns
    ("cube", 46, "ttp", 1e-6, 100, True, 0.5),      # two rows a thread, state held
])
def test_persistent_steps_match_single_launches(lib, cuda, mesh, size, model, tol, max_iter, guess, theta):
    steps = 120
    sim = _sim(mesh, size, model, cuda, theta, steps=steps)
    a = _run(sim, tol, max_iter, guess, 0, [steps])
    if mesh == "ico" and size == 6:
        assert sim.system.sell_dcol is None
    assert bool(sim.system.a_split) == (theta == 0.5)
    b = _run(sim, tol, max_iter, guess, 2, [steps])
    assert torch.equal(a["iters"], b["iters"])
    for k in ("x", "state"):
        # Mitchell-Schaeffer's gate switches branch at a voltage: a node on it may go either way for a step
        bound = 1e-2 if (k, model) == ("state", "ms") else steps * 2.0 ** -23
        err = (a[k] - b[k]).abs().max().item() / b[k].abs().max().item()
        assert err <= bound, (k, err)
    assert (a["at"] - b["at"]).abs().max().item() <= 0.0201 and (a["rt"] - b["rt"]).abs().max().item() <= 0.0201


@pytest.mark.parametrize("fused_step,kernel", [(-1, 2), (0, 1), (1, 2), (2, 1), (3, 2)])
def test_forms_of_a_single_step(lib, cuda, fused_step, kernel):
    """2 asks for two launches; every other value but 0 for the fused one, as before there was a 2."""
    sim = _sim("cube", 6, "ttp", cuda)
    sim.prepare(1e-6, 1e-6, 100, snapshot_interval=sim.T)
    sim.set_launch(fused_step=fused_step)
    assert lib.tcb_mono_cg_kernel(C.byref(sim._sim["struct"])) == kernel


def test_stretches_of_any_length_are_the_same(lib, cuda):
    """Where a launch begins and ends changes nothing, bit for bit: 145 steps at once
    (more than one launch's limit), and in stretches with and without the state held on chip."""
    sim = _sim("cube", 10, "ttp", cuda)
    ref = _run(sim, 1e-6, 100, True, 0, [145], frames=True)
    got = _run(sim, 1e-6, 100, True, 0, [1, 1, 2, 3, 4, 5, 129], frames=True)
    for k in ref:
        assert torch.equal(ref[k], got[k]), k


def test_step_graph_recorded_while_garbage_holds_device_memory(lib, cuda):
    """A collection in the middle of a recording would free what unreachable cycles hold
    (other step graphs, tensors) on the recording thread and break it: with the collector
    at its most eager the recording still succeeds."""
    import gc
    sim = _sim("cube", 5, "ms", cuda)
    sim.prepare(1e-5, 1e-5, 100, snapshot_interval=sim.T)
    old = gc.get_threshold()
    try:
        for _ in range(20):
            cycle = [torch.empty(3 << 20, device=cuda), sim.capture_steps(3)]
            cycle.append(cycle)
            del cycle
            gc.set_threshold(1, 1, 1)
            sim.capture_steps(5)()
            gc.set_threshold(*old)
    finally:
        gc.set_threshold(*old)
    torch.cuda.synchronize(cuda)


def test_first_steps_on_a_stream_of_the_callers(lib, cuda):
    """The first steps of a simulation on a stream other than the current one, which is busy:
    they neither wait for it nor read an exchange buffer that it has yet to zero, so they are those on
    the current stream bit for bit.  Freed memory of that size is full of ones."""
    sim = _sim("cube", 20, "ttp", cuda)
    ref = _run(sim, 1e-6, 100, True, 0, [20])
    nbytes = sim._sim["work"].numel()
    sim.prepare(1e-6, 1e-6, 100, snapshot_interval=sim.T)
    dirty = [torch.full((nbytes,), 255, device=cuda, dtype=torch.uint8) for _ in range(4)]
    big = torch.empty((2, 1 << 30), device=cuda, dtype=torch.uint8)
    side = torch.cuda.Stream(cuda)
    torch.cuda.synchronize(cuda)
    del dirty
    for _ in range(300):          # about 0.1 s
        big[1].copy_(big[0])
    busy = torch.cuda.Event()
    busy.record()
    assert sim.run_steps(12, stream=side) == 12
    class Handle:                 # any object with a stream's address, as stream_ptr takes
        cuda_stream = side.cuda_stream
    assert sim.run_steps(8, stream=Handle()) == 8
    side.synchronize()
    assert not busy.query()       # the steps did not wait for the copies
    assert sim._sim["work"] is not None
    torch.cuda.synchronize(cuda)
    assert torch.equal(sim._sim["x"][:, : sim.n_nodes], ref["x"])
    assert torch.equal(sim._sim["step_iters"], ref["iters"])


def test_steps_recorded_by_the_caller_right_after_prepare(lib, cuda):
    """run_steps under a recording of the caller's own allocates, copies and waits for nothing: the
    recorded steps are the ones launched one by one, and later steps run as stretches again."""
    sim = _sim("cube", 10, "ttp", cuda)
    ref = _run(sim, 1e-6, 100, True, 2, [10])
    sim.prepare(1e-6, 1e-6, 100, snapshot_interval=sim.T)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        assert sim.run_steps(10) == 10
    assert sim._sim["work"] is None
    graph.replay()
    torch.cuda.synchronize(cuda)
    assert torch.equal(sim._sim["x"][:, : sim.n_nodes], ref["x"])
    sim.run_steps(3)
    assert sim._sim["work"] is not None and int(sim._sim["counter"][0].item()) == 14


def test_launch_shape_taken_back_before_the_first_stretch(lib, cuda):
    """Steps under a pinned launch shape ask for no exchange buffer; without it the next ones do."""
    sim = _sim("cube", 6, "ms", cuda)
    sim.prepare(1e-6, 1e-6, 100, snapshot_interval=sim.T)
    sim.set_launch(fused_step=1)
    sim.run_steps(2)
    assert sim._sim["work"] is None
    sim.set_launch(fused_step=0)
    sim.run_steps(2)
    assert sim._sim["work"] is not None and int(sim._sim["counter"][0].item()) == 5


def test_replay_on_another_stream_follows_what_came_before_the_recording(lib, cuda):
    """Steps queued behind other work before the recording, replayed right after it on an idle stream
    that nothing orders with the first: the replay comes after them."""
    sim = _sim("cube", 20, "ttp", cuda)
    ref = _run(sim, 1e-6, 100, True, 0, [8])
    sim.prepare(1e-6, 1e-6, 100, snapshot_interval=sim.T)
    sim.run_steps(1)
    big = torch.empty((2, 1 << 30), device=cuda, dtype=torch.uint8)
    for _ in range(100):
        big[1].copy_(big[0])
    sim.run_steps(2)
    replay = sim.capture_steps(5)
    side = torch.cuda.Stream(cuda)
    with torch.cuda.stream(side):
        replay()
    side.synchronize()
    assert torch.equal(sim._sim["x"][:, : sim.n_nodes], ref["x"])
    assert torch.equal(sim._sim["step_iters"], ref["iters"])


FIRST_CALLS = """
import ctypes as C, threading, torch
from tests.test_gpu_steps import _sim
from torchcor_b200 import _lib
lib, cuda = _lib.load(), torch.device("cuda", 0)
sims = [_sim("cube", 12 + k % 3, "ttp", cuda) for k in range(12)]
for s in sims:
    s.prepare(1e-6, 1e-6, 100, snapshot_interval=s.T)
torch.cuda.synchronize()
together = threading.Barrier(len(sims))
asked, failed = [None] * len(sims), []
def work(s):
    n = C.c_int32()
    slices = _lib.ptr(s.system.host_slices)
    return lib.tcb_mono_work_bytes_host(C.byref(s._sim["struct"]), slices, C.byref(n)), n.value
def first(k):
    try:
        stream = torch.cuda.Stream()
        together.wait()
        asked[k] = work(sims[k])                 # the first questions about the device
        sims[k].run_steps(3, stream=stream)      # the first launches
        stream.synchronize()
        _lib.check(lib.tcb_mono_check(C.byref(sims[k]._sim["struct"]), stream.cuda_stream))
    except BaseException as e:
        failed.append(repr(e))
threads = [threading.Thread(target=first, args=(k,)) for k in range(len(sims))]
for t in threads: t.start()
for t in threads: t.join()
assert not failed, failed
assert asked == [work(s) for s in sims] and all(b > 0 for b, _ in asked), asked
for s in sims[3:]:
    ref = sims[sims.index(s) % 3]
    assert torch.equal(s._sim["x"], ref._sim["x"])
print("same")
"""


def test_first_calls_from_several_threads(lib, cuda):
    """The limits of a device and the kernels' attributes are set by whichever thread comes first;
    the others wait for the finished values."""
    import subprocess
    import sys
    from pathlib import Path
    root = Path(__file__).resolve().parent.parent
    r = subprocess.run([sys.executable, "-c", FIRST_CALLS], cwd=root, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "same" in r.stdout, r.stderr[-2000:]


@pytest.mark.parametrize("mesh,size,model,tol", [("cube", 20, "ms", 1e-8), ("cube", 12, "ttp", 1e-8), ("ico", 4, "crn", 1e-8),
                                                 ("cube", 20, "ttp", 1e-5), ("ico", 5, "ms", 1e-6)])
def test_every_stopping_test_ends_the_same_iterations(lib, cuda, monkeypatch, mesh, size, model, tol):
    """The streaming kernel sums |z'|^2 itself; the resident, the batched and the persistent kernels
    take it from the sums of the pass before (over z and w = D A p rounded to float32 in the
    first two).  Where a pass leaves 1e-3 of |z| that is right to about 1e-4 of it: the kernels stop
    at the same iteration in every step, tight tolerances and many passes a step included."""
    from torchcor_b200.simulator import MonodomainBatch
    steps = 60
    sim = _sim(mesh, size, model, cuda, steps=steps)
    iters = {"stretch": _run(sim, tol, 100, False, 0, [steps])["iters"],
             "resident": _run(sim, tol, 100, False, 2, [steps])["iters"],
             "fused": _run(sim, tol, 100, False, 1, [steps])["iters"]}
    for variant in (1, 2, 3):
        sim._sim = None
        batch = MonodomainBatch(cuda, max_sims=1)
        batch.add(sim, tol, tol, 100, linear_guess=False, snapshot_interval=sim.T)
        batch.set_cg(variant)
        batch.step(steps)
        batch.check()
        iters[f"batch{variant}"] = sim._sim["step_iters"].clone()
    monkeypatch.setenv("TCB_CG_KERNEL", "streaming")
    want = _run(sim, tol, 100, False, 2, [steps])["iters"]
    if tol < 1e-7:
        assert want.max().item() >= 4          # several passes a step
    for name, got in iters.items():
        assert torch.equal(got, want), (name, (got - want).nonzero().tolist())


def test_exchange_buffer_made_beside_outlives_steps_on_the_current_stream(lib, cuda):
    """First steps on a stream of the caller's, more behind other work on the current one, then the
    buffer is dropped: its memory is not handed out on the first stream while the steps are pending."""
    sim = _sim("cube", 20, "ttp", cuda)
    ref = _run(sim, 1e-6, 100, True, 0, [20])
    sim.prepare(1e-6, 1e-6, 100, snapshot_interval=sim.T)
    torch.cuda.synchronize(cuda)
    side = torch.cuda.Stream(cuda)
    sim.run_steps(10, stream=side)
    side.synchronize()
    big = torch.empty((2, 1 << 30), device=cuda, dtype=torch.uint8)
    for _ in range(100):
        big[1].copy_(big[0])
    sim.run_steps(10)
    done = torch.cuda.Event()
    done.record()
    d = sim._sim
    work = d.pop("work")
    at, nbytes = work.data_ptr(), work.numel()
    del work
    with torch.cuda.stream(side):
        others = [torch.full((nbytes,), 255, device=cuda, dtype=torch.uint8) for _ in range(4)]
    assert not done.query()
    assert at not in [t.data_ptr() for t in others]
    torch.cuda.synchronize(cuda)
    assert torch.equal(d["x"][:, : sim.n_nodes], ref["x"])

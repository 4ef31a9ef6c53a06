"""What handles choose for themselves, and what those of one process share or keep between calls: the
autotuner's team sizes, the captured steps (their own and a caller's), the step counter and the tables of a hook loop, the
runtime's record of an error."""
import time

import numpy as np
import pytest

from axisem3d_b200 import meshgen
from axisem3d_b200.solver import EngineError, Solver

pytestmark = pytest.mark.gpu


def test_a_failed_call_does_not_fail_the_next_one(built):
    """The legacy default stream (address 1) cannot be captured: a run on it is refused by the host
    side of the runtime. That error is reported once, not again by the next launch of this handle or
    of another one."""
    m = meshgen.cartesian_model(nx=7, nz=5, nr=5)
    with Solver(m, "fp64") as a, Solver(m, "fp64") as b:
        b.run(4)
        a.set_stream(1)
        with pytest.raises(EngineError, match="BeginCapture"):
            a.run(4)
        b.run(4)
        a.set_stream(None)
        a.run(8)
        d, e = a.get_field("displ"), b.get_field("displ")
    # the atomic sums of 8 steps in another order
    assert np.linalg.norm(d - e) <= 1e-13 * np.linalg.norm(e)


def _captured_stiffness(s, *buffers):
    """One no-allocation stiffness evaluation of the device buffers x, f (and of the fluid's) as a
    captured graph of the caller's stream."""
    import torch
    stream = torch.cuda.Stream()
    s.set_stream(stream.cuda_stream)
    torch.cuda.synchronize()
    ptr = [b.data_ptr() for b in buffers]
    s.compute_stiffness_noalloc(*ptr)      # looks the library's array up
    stream.synchronize()
    g = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(g, stream=stream):
        s.compute_stiffness_noalloc(*ptr)
    return g, stream


def _on_device(u, dtype):
    import torch
    return torch.view_as_real(torch.from_numpy(u).to("cuda", dtype)).contiguous()


def _block_threads(s, u):
    """Threads per block of the kernels of one stiffness evaluation, from a captured graph of it."""
    import torch
    from cuda.bindings import driver
    x = _on_device(u, torch.complex128)
    g, stream = _captured_stiffness(s, x, torch.zeros_like(x))
    graph = driver.CUgraph(g.raw_cuda_graph())
    count = driver.cuGraphGetNodes(graph)[2]
    threads = []
    for node in driver.cuGraphGetNodes(graph, count)[1]:
        if driver.cuGraphNodeGetType(node)[1] == driver.CUgraphNodeType.CU_GRAPH_NODE_TYPE_KERNEL:
            threads.append(int(driver.cuGraphKernelNodeGetParams(node)[1].blockDimX))
    s.set_stream(None)
    return threads


def test_autotuner_keeps_the_large_blocks(built):
    """The 512-thread block of large 3-D elements is 1.5 times as fast as 256 threads here, so an
    autotuned handle must end with it like a plain one does."""
    m = meshgen.microbench_model(n_elem=400, nr_choices=[75], rheology="iso", attenuation=None, seed=2)
    u = meshgen.random_displacement(m, seed=4)
    with Solver(m, "fp64") as s:
        assert _block_threads(s, u) == [512]
    with Solver(m, "fp64", team_sizes={4: 256}) as s:
        assert _block_threads(s, u) == [256]
    with Solver(m, "fp64", autotune=True) as s:
        assert _block_threads(s, u) == [512]


@pytest.mark.parametrize("pieces", [[300], [20] * 15, [100, 100, 100], [8, 255, 1, 7, 9, 20], [250, 8, 42]])
def test_graph_of_several_steps_behind_single_ones(built, pieces):
    """The graph of eight steps is made once a handle has been asked for 256 steps, behind queued
    single ones; source and record tables grow between the runs and both graphs follow them."""
    m = meshgen.cartesian_model(nx=5, nz=4, nr=5, nstations=3, record_interval=7)
    with Solver(m, "fp64") as s:
        s.run(300, graph=False)
        ref, seis = s.get_field("displ"), s.seismograms()
    with Solver(m, "fp64") as s:
        for n in pieces:
            s.run(n)
        assert s.step == 300
        d, g = s.get_field("displ"), s.seismograms()
    # the order of the atomic sums, over 300 steps
    assert np.linalg.norm(d - ref) <= 1e-11 * np.linalg.norm(ref)
    assert g.shape == seis.shape and np.linalg.norm(g - seis) <= 1e-11 * np.linalg.norm(seis)


def test_graph_of_several_steps_in_a_first_run(built):
    """On a mesh whose steps cover the building, a first run of 20 steps has the graph of eight too."""
    m = meshgen.microbench_model(n_elem=1500, nr_choices=[40], rheology="iso", attenuation="full", seed=6)
    u = meshgen.random_displacement(m, seed=4)
    out = []
    for graph in (False, True):
        with Solver(m, "fp64") as s:
            s.set_field(u, "displ")
            for n in (20, 13):
                s.run(n, graph=graph)
            assert s.step == 33
            out.append(s.get_field("displ"))
    assert np.linalg.norm(out[1] - out[0]) <= 1e-11 * np.linalg.norm(out[0])


def test_short_runs_do_not_pay_for_graphs(built):
    """Runs of 20 steps of a new handle, the tables growing under them, take no longer than twice
    their launches one by one (three to four times with graphs of eight steps made for each)."""
    m = meshgen.cartesian_model(nx=40, nz=40, nr=5, nstations=20)
    best = {}
    for graph in (False, True) * 8:
        with Solver(m, "fp32") as s:
            s.run(20, graph=graph)
            s.synchronize()
            t = time.perf_counter()
            for _ in range(2):
                s.run(20, graph=graph)
                s.synchronize()
            best[graph] = min(best.get(graph, 1.0), time.perf_counter() - t)
    assert best[True] <= 2 * best[False], best


def _hooks(s, t):
    s.apply_sources(t)
    s.compute_stiffness()
    s.apply_bc_before_assembly()
    s.record_stations(t)
    s.apply_bc_after_assembly()
    s.stiff_to_accel()
    s.newmark_update()


def test_hooks_queue_steps_while_the_tables_grow(built):
    """A hook loop that nothing waits in, from an empty source table: each growth gives the old
    table back only when the queued steps have read it."""
    m = meshgen.cartesian_model(nx=12, nz=9, nr=5, nstations=3)
    with Solver(m, "fp64") as s:
        s.run(200)
        ref = s.get_field("displ")
    with Solver(m, "fp64") as s:
        for t in range(200):
            _hooks(s, t)
        d = s.get_field("displ")
    assert np.linalg.norm(d - ref) <= 1e-11 * np.linalg.norm(ref)


def test_hooks_runs_and_streams_in_turn(built):
    """The device's step counter is set only when it does not hold the step already: hooks before and
    after a run, a repeated step and a change of stream each record and shake the step they are given."""
    import torch
    n, interval = 24, 2
    m = meshgen.cartesian_model(nx=6, nz=5, nr=5, nstations=4, record_interval=interval)
    u0, other = (meshgen.random_displacement(m, seed=k) * 1e-3 for k in (9, 10))
    with Solver(m, "fp64") as s:
        s.set_field(u0, "displ")
        s.run(n)
        ref, seis = s.get_field("displ"), s.seismograms()
    stream = torch.cuda.Stream()
    with Solver(m, "fp64") as s:
        # records of another wavefield in every slot, so that one left out shows
        s.set_field(other, "displ")
        s.run(n)
        assert np.linalg.norm(s.seismograms() - seis) > 0.1 * np.linalg.norm(seis)
        zero = np.zeros_like(u0)
        for name, v in (("displ", u0), ("veloc", zero), ("accel", zero), ("stiff", zero)):
            s.set_field(v, name)
        for t in range(n):
            _hooks(s, t)
            if t in (5, 6, 15):
                # a run elsewhere in time, then the fields as they were
                keep = {k: s.get_field(k) for k in ("displ", "veloc", "accel", "stiff")}
                k0 = s.step
                s.run(3 if t == 15 else t)
                assert s.step > k0
                for k, v in keep.items():
                    s.set_field(v, k)
            if t == 10:
                s.synchronize()
                s.set_stream(stream.cuda_stream)
            if t == 18:
                s.synchronize()
                s.set_stream(None)
        d, g = s.get_field("displ"), s.seismograms()
    assert np.linalg.norm(d - ref) <= 1e-12 * np.linalg.norm(ref)
    assert np.linalg.norm(g[:seis.shape[0]] - seis) <= 1e-12 * np.linalg.norm(seis)


def test_adjoint_after_checkpoints_that_did_not_fit(built):
    """Checkpoints beyond the GPU's memory are refused, and the run before them, whose checkpoints gave
    way, cannot be gone back over."""
    from axisem3d_b200 import _lib as L
    m = meshgen.cartesian_model(nx=8, nz=8, nr=9, nstations=2, record_interval=10 ** 6)
    with Solver(m, "fp64") as s:
        s.forward_checkpointed(4, 2)
        seis = s.seismograms()
        n = int(4e11 / (16 * s.field_size()))          # 400 GB of displacement alone
        with pytest.raises(EngineError) as ei:
            s.forward_checkpointed(n, 1)
        assert ei.value.code == L.AXG_E_NOMEM
        with pytest.raises(EngineError) as ei:
            s.adjoint(seis)
        assert ei.value.code == L.AXG_E_STATE
        s.forward_checkpointed(4, 2)
        g = s.adjoint(s.seismograms())
    assert np.all(np.isfinite(g["moduli"]))


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_captured_stiffness_of_several_buckets(built, precision):
    """A caller's capture takes the branches of every bucket, solid and fluid, into its graph; a replay
    on other inputs in the same buffers gives the handle's own stiffness."""
    import torch
    m = meshgen.spherical_model(n_theta=24, n_solid_layers=6, n_fluid_layers=2, nr_max=40)
    dtype = torch.complex128 if precision == "fp64" else torch.complex64
    us, uf = meshgen.random_displacement(m, seed=5), meshgen.random_displacement(m, seed=6, solid=False)
    with Solver(m, precision) as s:
        s.set_field(us, "displ")
        s.set_field(uf, "displ", solid=False)
        s.compute_stiffness()
        ref = s.get_field("stiff"), s.get_field("stiff", solid=False)
    with Solver(m, precision) as s:
        x, y = _on_device(0 * us, dtype), _on_device(0 * uf, dtype)
        f, h = torch.zeros_like(x), torch.zeros_like(y)
        g, stream = _captured_stiffness(s, x, f, y, h)
        x.copy_(_on_device(us, dtype))
        y.copy_(_on_device(uf, dtype))
        for _ in range(2):
            f.zero_()
            h.zero_()
            torch.cuda.synchronize()
            with torch.cuda.stream(stream):
                g.replay()
            torch.cuda.synchronize()
        got = [torch.view_as_complex(t).cpu().numpy() for t in (f, h)]
        s.set_stream(None)
    for a, b in zip(got, ref):
        assert np.linalg.norm(a.ravel() - b) <= (1e-12 if precision == "fp64" else 1e-6) * np.linalg.norm(b)


def test_a_handle_that_cannot_be_made_keeps_its_model(built):
    """axg_finalize takes the model over; refused (modes that no block holds), it is refused again and
    not made of an empty one."""
    from axisem3d_b200 import _lib as L

    class Unchecked(Solver):
        def _check(self, rc):
            self.rc = rc

    m = meshgen.microbench_model(n_elem=2, nr_choices=[260], rheology="iso", attenuation=None)
    s = Unchecked(m, "fp64")
    assert s.rc == L.AXG_E_UNSUPPORTED
    assert s.lib.axg_finalize(s.h) == L.AXG_E_UNSUPPORTED
    assert b"too large" in s.lib.axg_last_error(s.h)
    assert s.lib.axg_run(s.h, 1, 1) == L.AXG_E_STATE
    s.close()


def test_refused_hooks_leave_a_capture_alone(built):
    """The hooks that set the step, and runs, are refused while the caller's stream is capturing, also
    where they would have to grow a table first; the capture goes on and its graph is whole."""
    import torch
    m = meshgen.cartesian_model(nx=6, nz=5, nr=5, nstations=2)
    u = meshgen.random_displacement(m, seed=9)
    with Solver(m, "fp64") as s:
        s.set_field(u, "displ")
        s.compute_stiffness()
        ref = s.get_field("stiff")
    with Solver(m, "fp64") as s:
        x = _on_device(u, torch.complex128)
        f = torch.zeros_like(x)
        stream = torch.cuda.Stream()
        s.set_stream(stream.cuda_stream)
        torch.cuda.synchronize()
        s.compute_stiffness_noalloc(x.data_ptr(), f.data_ptr())
        stream.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=stream, capture_error_mode="thread_local"):
            s.compute_stiffness_noalloc(x.data_ptr(), f.data_ptr())
            for call in (lambda: s.apply_sources(100), lambda: s.record_stations(100), lambda: s.run(20)):
                with pytest.raises(EngineError, match="capturing"):
                    call()
        f.zero_()
        torch.cuda.synchronize()
        with torch.cuda.stream(stream):
            g.replay()
        torch.cuda.synchronize()
        got = torch.view_as_complex(f).cpu().numpy().ravel()
        s.set_stream(None)
        s.run(4)
    assert np.linalg.norm(got - ref) <= 1e-12 * np.linalg.norm(ref)

"""Work buffers of captured _dev calls: a graph keeps its own for as long as it
can be launched, whatever later calls do on the streams it was captured on."""
import gc

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


class Dt:
    """dt_ng of ncol columns, its fields and result on the device."""

    def __init__(self, pkg, nk, ncol, seed):
        import torch
        F, self.C = pkg.synth.dt_inputs(nk, ncol, 0.25, seed)
        self.pkg, self.nk, self.ncol, self.ld = pkg, nk, ncol, pkg.batch.pad_ld(ncol)
        grid = type("G", (), dict(nk=nk, ncol=ncol, ld=self.ld))()
        self.F = pkg.dynamics._dev_fields(F, grid, ("expz", "dift"), "cuda")
        self.out = torch.zeros((nk, self.ld), dtype=torch.float64, device="cuda")
        self.status = torch.full((1,), -1, dtype=torch.int32, device="cuda")

    def issue(self, st):
        self.pkg.dt_ng_dev(self.F, self.C, self.out, self.nk, self.ncol, self.ld, status=self.status, stream=st)

    def capture(self, st):
        import torch
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=st, capture_error_mode="thread_local"):
            self.issue(st)
        return g

    def result(self, st, run):
        import torch
        self.out.fill_(float("nan"))
        self.status.fill_(-1)
        torch.cuda.synchronize()
        with torch.cuda.stream(st):
            run()
        torch.cuda.synchronize()
        assert int(self.status.item()) == self.pkg.TG_OK
        return self.out[:, :self.ncol].clone()


def bits(a, b):
    import torch
    return torch.equal(a.view(torch.int64), b.view(torch.int64))


@pytest.mark.parametrize("eager_on_the_stream", [True, False])
def test_growth_and_eviction_leave_a_graph_alone(cuda, pkg, eager_on_the_stream):
    import torch
    st = torch.cuda.Stream()
    other = st if eager_on_the_stream else torch.cuda.Stream()
    small, large = Dt(pkg, 57, 700, 1), Dt(pkg, 57, 9000, 2)
    want = small.result(other, lambda: small.issue(other))
    g = small.capture(st)
    assert bits(small.result(st, g.replay), want)
    large.result(st, lambda: large.issue(st))             # the stream's own buffers grow
    assert bits(small.result(st, g.replay), want)
    for _ in range(20):                                   # more streams than there are workspaces
        s = torch.cuda.Stream()
        large.result(s, lambda: large.issue(s))
    hold = torch.full((1 << 24,), float("nan"), dtype=torch.float64, device="cuda")
    assert bits(small.result(st, g.replay), want) and bool(hold.isnan().all())


def test_graphs_of_one_stream_run_side_by_side(cuda, pkg):
    import torch
    st, a, b = torch.cuda.Stream(), torch.cuda.Stream(), torch.cuda.Stream()
    p, q = Dt(pkg, 57, 6000, 3), Dt(pkg, 57, 6000, 4)
    want = [x.result(st, lambda: x.issue(st)) for x in (p, q)]
    gp, gq = p.capture(st), q.capture(st)
    for x in (p, q):
        x.out.fill_(float("nan"))
    torch.cuda.synchronize()
    for _ in range(40):
        with torch.cuda.stream(a):
            gp.replay()
        with torch.cuda.stream(b):
            gq.replay()
    torch.cuda.synchronize()
    for x, w in zip((p, q), want):
        assert bits(x.out[:, :x.ncol], w)


def test_column_layout_solve_keeps_its_relayout(cuda, pkg, orc):
    import torch
    st = torch.cuda.Stream()
    sysm = pkg.synth.scalar_system(29, 500, 0.5, 7, d0_range=(1e-3, 1e-2), loss=("uniform", 0.0, 1e-3))
    want = orc.trsolv_ng(*[np.asfortranarray(v) for v in sysm], 29)
    dev = [torch.from_numpy(np.ascontiguousarray(v.T)).cuda() for v in sysm]
    x = torch.zeros_like(dev[3])
    solve = lambda d, out, n: pkg.trsolv_dev(*d, out, 29, 29, n, layout=pkg.TG_LAYOUT_COLUMN, stream=st)  # noqa: E731
    with torch.cuda.stream(st):
        solve(dev, x, 500)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=st, capture_error_mode="thread_local"):
        solve(dev, x, 500)
    big = [v.repeat(40, 1) for v in dev]
    with torch.cuda.stream(st):
        solve(big, torch.zeros_like(big[3]), 20000)
        x.fill_(float("nan"))
        g.replay()
    torch.cuda.synchronize()
    assert np.array_equal(x.cpu().numpy().T, want)


def test_buffers_of_destroyed_graphs_are_used_again(cuda, pkg):
    """60 graphs, one alive at a time: the rows of 20,000 columns are 36 MB a graph."""
    import torch
    st, d = torch.cuda.Stream(), Dt(pkg, 57, 20000, 5)
    want = d.result(st, lambda: d.issue(st))
    free = []
    for i in range(60):
        g = d.capture(st)
        if i % 20 == 19:
            assert bits(d.result(st, g.replay), want)
        del g
        gc.collect()
        torch.cuda.synchronize()
        free.append(torch.cuda.mem_get_info()[0])
    assert free[9] - free[-1] <= 20 * 37e6


def test_owned_captures(cuda, pkg):
    """60 graphs whose owner says when they are gone; the refusals."""
    import torch
    st, d = torch.cuda.Stream(), Dt(pkg, 57, 20000, 6)
    want = d.result(st, lambda: d.issue(st))
    with pytest.raises(pkg.TgError):          # no capture
        pkg.capture_own(st)
    with pytest.raises(pkg.TgError):          # nobody's
        pkg.capture_release(1 << 60)
    free = []
    for i in range(60):
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=st, capture_error_mode="thread_local"):
            own = pkg.capture_own(st)
            d.issue(st)
            with pytest.raises(pkg.TgError):  # too late
                pkg.capture_own(st)
        if i % 20 == 19:
            assert bits(d.result(st, g.replay), want)
        g.reset()
        pkg.capture_release(own)
        assert bits(d.result(st, lambda: d.issue(st)), want)
        free.append(torch.cuda.mem_get_info()[0])
    with pytest.raises(pkg.TgError):          # given back already
        pkg.capture_release(own)
    assert free[9] - free[-1] <= 8 * 37e6


def test_steps_of_two_sizes(cuda, pkg):
    """Steps captured one after another on one stream, the larger one later,
    more of them than the library has workspaces; then each replayed."""
    import torch
    dyn, st, steps, want = pkg.dynamics, torch.cuda.Stream(), [], []
    for i, (nlon, nlat) in enumerate([(9, 5), (30, 20), (12, 7), (40, 22), (9, 5)]):
        grid = dyn.Grid(29, nlon, nlat, 0.5, lat0_deg=20.0, dlat_deg=0.3)
        s = dyn.DynamicsStep(grid, dyn.synthetic_inputs(grid, 50 + i, nstep_sub=2))
        s.issue(st)
        torch.cuda.synchronize()
        want.append({k: v[:, :grid.ncol].clone() for k, v in s.outputs().items()})
        s.capture(st)
        steps.append(s)
    for s, w in zip(steps, want):
        for v in s.outputs().values():
            v.fill_(float("nan"))
        torch.cuda.synchronize()
        s.replay(st)
        torch.cuda.synchronize()
        for k, v in s.outputs().items():
            assert bits(v[:, :s.grid.ncol].contiguous(), w[k].contiguous()), k


def test_released_captures_without_eager_calls(cuda, pkg):
    """A caller that only captures and releases, 40 times."""
    import torch
    st, d = torch.cuda.Stream(), Dt(pkg, 57, 20000, 7)
    want, free = d.result(st, lambda: d.issue(st)), []
    for i in range(40):
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=st, capture_error_mode="thread_local"):
            own = pkg.capture_own(st)
            d.issue(st)
        assert bits(d.result(st, g.replay), want)
        g.reset()
        pkg.capture_release(own)
        free.append(torch.cuda.mem_get_info()[0])
    assert free[9] - free[-1] <= 8 * 37e6


def test_an_owned_graph_and_eager_calls_after_it(cuda, pkg):
    """The graph took over its stream's buffers: eager calls there get others."""
    import torch
    st = torch.cuda.Stream()
    p, q = Dt(pkg, 57, 6000, 8), Dt(pkg, 57, 6000, 9)
    want = [x.result(st, lambda: x.issue(st)) for x in (p, q)]
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=st, capture_error_mode="thread_local"):
        own = pkg.capture_own(st)
        p.issue(st)
    other = torch.cuda.Stream()
    for _ in range(20):
        with torch.cuda.stream(other):
            g.replay()
        q.issue(st)
    torch.cuda.synchronize()
    for x, w in zip((p, q), want):
        assert bits(x.out[:, :x.ncol], w)
    g.reset()
    pkg.capture_release(own)


def test_captures_beside_other_threads(cuda, pkg):
    """Three threads, each on its stream: eager calls, captures (owned and not),
    replays, releases.  What one thread's graphs leave, the others' calls take."""
    import threading
    import torch
    sizes, errs, lock, start = (700, 3000, 1500), [], threading.Lock(), threading.Barrier(3)
    work = [[Dt(pkg, 57, n, 20 + i) for i, n in enumerate(sizes)] for _ in range(3)]
    streams = [torch.cuda.Stream() for _ in range(3)]
    want = [d.result(streams[0], lambda: d.issue(streams[0])) for d in work[0]]
    for st, ds in zip(streams, work):          # a growing call synchronises, which another thread's capture does not survive
        ds[1].result(st, lambda: ds[1].issue(st))

    def run(t):
        try:
            st = streams[t]
            start.wait()
            for it in range(9):
                d, w = work[t][(t + it) % 3], want[(t + it) % 3]
                with torch.cuda.stream(st):
                    for _ in range(3):
                        d.issue(st)
                g, own = torch.cuda.CUDAGraph(), None
                with lock:                     # torch's own bookkeeping of captures
                    with torch.cuda.graph(g, stream=st, capture_error_mode="thread_local"):
                        own = pkg.capture_own(st) if it % 2 else None
                        d.issue(st)
                with torch.cuda.stream(st):
                    d.out.fill_(float("nan"))
                    g.replay()
                    r = d.out[:, :d.ncol].clone()
                st.synchronize()
                if not bits(r, w):
                    errs.append((t, it))
                with lock:
                    g.reset()
                if own is not None:
                    pkg.capture_release(own)
        except Exception as e:                 # reported below, with the thread's number
            errs.append((t, repr(e)))

    threads = [threading.Thread(target=run, args=(t,)) for t in range(3)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert errs == []

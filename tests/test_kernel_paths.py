"""The solve kernels' size-dependent paths against the CPU oracle, bit for
bit (fp64), at the sizes where a path starts, ends or changes."""
import numpy as np
import pytest

from odevec_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _solver(S, wl, **kw):
    kw.setdefault("precision", "fp64")
    kw.setdefault("nvector", wl.group)
    ode = S.Odevec(wl.network, RelativeTolerance=wl.rtol, AbsoluteTolerance=wl.atol, MinimalTimestep=wl.dt_min,
                   raise_on_failure=False, **kw)
    S.InitOdevec(ode)
    return ode


def _gpu(S, ode, wl, mask=None):
    import torch
    y = torch.tensor(wl.y, device="cuda")
    t, dt = S.SolveODE(ode, torch.tensor(wl.t0, device="cuda"), torch.tensor(wl.dt0, device="cuda"),
                       torch.tensor(wl.t_stop, device="cuda"), y, Mask=mask)
    torch.cuda.synchronize()
    return [a.cpu().numpy() for a in (y, t, dt, ode.status, ode.stats)]


def _oracle(O, wl, group=None, **kw):
    return O.solve(wl.network, wl.y, wl.t0, wl.dt0, wl.t_stop, wl.rtol, wl.atol, wl.dt_min,
                   group=wl.group if group is None else group, **kw)


def _same(g, o):
    for name, a, b in zip(("y", "t", "dt", "status", "stats"), g, o):
        assert np.array_equal(a, b, equal_nan=a.dtype.kind == "f"), "%s differs in %d places" % (name, int(np.sum(np.asarray(a) != np.asarray(b))))


def test_rate_table_sizes(gpu_lib, oracle):
    """Solves below, at and above the size from which the rates come from a
    table, on one solver whose table grows in between."""
    wls = {n: W.primordial(ncells=n, seed=20 + n % 7) for n in (4095, 4096, 9001)}
    ode = _solver(gpu_lib, wls[4096])
    try:
        for n in (4095, 4096, 9001, 4096):
            _same(_gpu(gpu_lib, ode, wls[n]), _oracle(oracle, wls[n]))
    finally:
        gpu_lib.CloseOdevec(ode)


@pytest.mark.parametrize("n", [1, 31, 148, 149, 593, 18944, 18945])
def test_few_cells_shapes(gpu_lib, oracle, n):
    """Launches of few cells: one lane of one warp, one warp per SM, a second
    warp on an SM, several lanes per warp, the last size of the rule and the
    first beyond it."""
    wl = W.orego(ncells=n, seed=3)
    wl.t_stop *= 0.05
    ode = _solver(gpu_lib, wl)
    try:
        _same(_gpu(gpu_lib, ode, wl), _oracle(oracle, wl))
    finally:
        gpu_lib.CloseOdevec(ode)


@pytest.mark.parametrize("groups", [1, 148, 149, 592, 593])
def test_few_groups_shapes(gpu_lib, oracle, groups):
    """The same for lockstep groups of 32 cells, a warp each."""
    wl = W.rober(ncells=32 * groups, seed=5)
    ode = _solver(gpu_lib, wl)
    try:
        _same(_gpu(gpu_lib, ode, wl), _oracle(oracle, wl))
    finally:
        gpu_lib.CloseOdevec(ode)


@pytest.mark.parametrize("n,mask,neg", [(1, False, False), (33, True, False), (149, False, True), (4737, True, True)])
def test_block_kernel(gpu_lib, oracle, n, mask, neg):
    """A large network, eight warps per 32 cells: one cell, a second block,
    more cells than SMs, more than all blocks hold; masked cells and
    CheckNegatives; then a continuation from the kept state."""
    import torch
    S = gpu_lib
    wl = W.syn64(ncells=n, seed=4)
    wl.t_stop[:] = 10.0 ** np.random.default_rng(2).uniform(-3.0, 3.0, n)
    m = None
    if mask:
        m = np.random.default_rng(1).random(n) > 0.2
        m[0] = True
    ode = _solver(S, wl, CheckNegatives=neg, staging=18)
    try:
        y = torch.tensor(wl.y, device="cuda")
        ws = S.Workspace(ode, n)
        ows = oracle.workspace(wl.network, n)
        oy, ot, od = wl.y, wl.t0, wl.dt0
        t, d = torch.tensor(wl.t0, device="cuda"), torch.tensor(wl.dt0, device="cuda")
        for k, resume in enumerate((False, True, "en_old")):
            ts = wl.t_stop * 2.0 ** k
            t, d = S.SolveODE(ode, t, d, torch.tensor(ts, device="cuda"), y, Mask=m, workspace=ws, resume=resume)
            torch.cuda.synchronize()
            oy, ot, od, ost, ostats = oracle.solve(wl.network, oy, ot, od, ts, wl.rtol, wl.atol, wl.dt_min, group=1,
                                                   mask=m, check_negatives=neg, ws=ows, resume=resume)
            _same([a.cpu().numpy() for a in (y, t, d, ode.status, ode.stats)], (oy, ot, od, ost, ostats))
    finally:
        S.CloseOdevec(ode)


@pytest.mark.parametrize("precision", ["fp64_fma", "fp32_lu"])
def test_block_kernel_forms(gpu_lib, precision):
    """The contracted forms give the bits of a thread per cell (staging 15)."""
    wl = W.syn64(ncells=300, seed=9)
    got = []
    for staging in (18, 15):
        ode = _solver(gpu_lib, wl, precision=precision, staging=staging, escalation=False)
        try:
            got.append(_gpu(gpu_lib, ode, wl))
        finally:
            gpu_lib.CloseOdevec(ode)
    _same(got[0], got[1])


@pytest.mark.parametrize("cells", [(32, 1, 1), (4096, 5000, 40), (33, 70, 700)])
def test_multi_block_jobs(gpu_lib, oracle, cells):
    """Several networks in one launch with blocks that go from one job's kernel
    to another's in either order."""
    import torch
    from odevec_b200.multi import SolveMany
    S = gpu_lib
    wls = [W.rober(cells[0], seed=2), W.primordial(cells[1], seed=2), W.syn64(cells[2], seed=2)]
    wls[2].t_stop[:] = 1e2
    odes, jobs = [], []
    for wl in wls:
        ode = _solver(S, wl, nvector=1)
        odes.append(ode)
        jobs.append((ode, *[torch.tensor(a, device="cuda") for a in (wl.t0, wl.dt0, wl.t_stop, wl.y)]))
    try:
        status = SolveMany(jobs, fused=True).run()
        torch.cuda.synchronize()
        for wl, job, st in zip(wls, jobs, status):
            o = _oracle(oracle, wl, group=1)
            _same([a.cpu().numpy() for a in (job[4], job[1], job[2], st)], o[:4])
    finally:
        for ode in odes:
            S.CloseOdevec(ode)


@pytest.mark.parametrize("n,shift", [(1, 0), (2, 0), (511, 0), (512, 0), (514, 0), (514, 1), (1025, 1)])
@pytest.mark.parametrize("in_place", [False, True])
def test_convert_widths(gpu_lib, oracle, n, shift, in_place):
    """Even and odd cell counts, arrays that do not start on 16 bytes, blocks
    that end inside a pair, the output over the input."""
    import torch
    from odevec_b200 import driver as D
    rng = np.random.default_rng(n)
    x = 10.0 ** rng.uniform(-20.0, 0.0, (16, n))
    rho = 10.0 ** rng.uniform(-26.0, -18.0, n)
    buf = torch.zeros(16 * n + 1, dtype=torch.float64, device="cuda")
    a = buf[shift:shift + 16 * n].view(16, n)
    r = torch.tensor(rho, device="cuda")
    for direction in (D.OV_X2N, D.OV_N2X):
        a.copy_(torch.tensor(x))
        out = D.convert("PRIMORDIAL_CSC_FF", a, r, direction, out=a if in_place else None)
        assert np.array_equal(out.cpu().numpy(), oracle.convert("PRIMORDIAL_CSC_FF", x, rho, direction))


@pytest.mark.parametrize("group,scale", [(1, 1e-9), (1, 1e4), (32, 1.0)])
def test_small_network_far_operands(gpu_lib, oracle, group, scale):
    """Three species: states far below and above the usual range (zeros among
    them), whose divisions leave or approach the range of the branch-free
    quotients."""
    wl = W.rober(ncells=96, seed=8)
    wl.y *= scale
    wl.y[:, ::5] *= 1e-290
    wl.y[1, ::3] = 0.0
    wl.t_stop[:] = 1e2
    ode = _solver(gpu_lib, wl, nvector=group, max_attempts=3000)
    try:
        _same(_gpu(gpu_lib, ode, wl), _oracle(oracle, wl, group=group, max_attempts=3000))
    finally:
        gpu_lib.CloseOdevec(ode)


@pytest.mark.parametrize("network", ["PRIMORDIAL_CSC_FF", "PRIMORDIAL_DENSE_NONE"])
@pytest.mark.parametrize("n", [1, 593, 18944, 18945])
def test_few_cells_on_chip(gpu_lib, oracle, network, n):
    """The shape of solves of few cells with the factors in shared memory: one
    lane, several lanes per warp, every lane once, and lanes that take a second
    cell."""
    wl = W.primordial(ncells=n, seed=6, network=network)
    wl.t_stop[:] = 1e8
    ode = _solver(gpu_lib, wl)
    try:
        _same(_gpu(gpu_lib, ode, wl), _oracle(oracle, wl))
    finally:
        gpu_lib.CloseOdevec(ode)


def test_few_cells_fp32_factors(gpu_lib):
    """FP32 factors of every network above four species: the same bits as in a
    shape that the caller fixes."""
    for wl in (W.hctoy(ncells=700, seed=3), W.primordial(ncells=700, seed=3)):
        wl.t_stop[:] = 1e8
        got = []
        for kw in ({}, {"staging": 3, "grid_blocks": 40}):
            ode = _solver(gpu_lib, wl, precision="fp32_lu", escalation=False, **kw)
            try:
                got.append(_gpu(gpu_lib, ode, wl))
            finally:
                gpu_lib.CloseOdevec(ode)
        _same(got[0], got[1])


@pytest.mark.parametrize("n", [75775, 75776])
def test_block_kernel_limit(gpu_lib, oracle, n):
    """The last cell count of the block kernel in FP64 and the first of a thread
    per cell."""
    wl = W.syn64(ncells=n, seed=12)
    wl.t_stop[:] = 1e-6
    ode = _solver(gpu_lib, wl)
    try:
        _same(_gpu(gpu_lib, ode, wl), _oracle(oracle, wl))
    finally:
        gpu_lib.CloseOdevec(ode)


@pytest.mark.parametrize("far", ["tiny", "nan", "masked"])
def test_lockstep_difference_quotients_far_operands(gpu_lib, oracle, far):
    """A lockstep group of a small network with difference quotients, one cell
    of which needs IEEE divisions: the whole group forms its matrix again (the
    quotients take a norm over the group), an ordinary group beside it does
    not."""
    wl = W.rober(ncells=64, seed=8, network="ROBER_DENSE_NONE_LU3")
    wl.y[:, 5] = (1e-290, 1e-295, 0.0) if far == "tiny" else np.nan
    wl.t_stop[:] = 1e2
    mask = np.ones(64, dtype=bool)
    mask[5] = far != "masked"
    ode = _solver(gpu_lib, wl, max_attempts=3000)
    try:
        _same(_gpu(gpu_lib, ode, wl, mask), _oracle(oracle, wl, max_attempts=3000, mask=mask))
    finally:
        gpu_lib.CloseOdevec(ode)


@pytest.mark.parametrize("options", [dict(max_attempts=40), dict(CheckNegatives=True), dict(fix_restart=True)])
def test_block_kernel_exits(gpu_lib, oracle, options):
    """The block kernel's ways out of a cell, and its restarts at order 1: cells
    out of attempts, steps below dt_min after a negative prediction and after a
    Newton failure (a NaN and an infinite state), beside ordinary cells."""
    wl = W.syn64(ncells=70, seed=4)
    wl.t_stop[:] = 10.0 ** np.random.default_rng(2).uniform(-3.0, 3.0, 70)
    wl.y[7, 3], wl.y[5, 40], wl.y[9, 66] = np.nan, -1e-3, np.inf
    ode = _solver(gpu_lib, wl, staging=18, **options)
    try:
        kw = {"check_negatives" if k == "CheckNegatives" else k: v for k, v in options.items()}
        _same(_gpu(gpu_lib, ode, wl), _oracle(oracle, wl, **kw))
    finally:
        gpu_lib.CloseOdevec(ode)


@pytest.mark.parametrize("precision,max_attempts", [("fp64", 0), ("fp32_lu", 0), ("fp32_lu", 5)])
def test_block_kernel_yields(gpu_lib, precision, max_attempts):
    """The block kernel stops starting cells, and continuations start the rest,
    the escalation of failed cells (with five attempts: all of them) included:
    the bits of one uninterrupted solve.  More cells than all blocks hold."""
    import torch
    S = gpu_lib
    n = 6000
    wl = W.syn64(ncells=n, seed=5)
    wl.t_stop[:] = 1e2
    got = []
    for yielding in (False, True):
        ode = _solver(S, wl, precision=precision, max_attempts=max_attempts)
        try:
            y, t, d, ts = (torch.tensor(a, device="cuda") for a in (wl.y, wl.t0, wl.dt0, wl.t_stop))
            st = torch.zeros(n, dtype=torch.int32, device="cuda")
            flag = torch.ones(1, dtype=torch.int32, device="cuda")
            S.set_yield(ode, flag if yielding else None)
            S.SolveODERange(ode, 0, n, t, d, ts, y, st)
            if yielding:
                assert S.cells_started(ode) < n
                for _ in range(20):
                    S.SolveODERange(ode, 0, n, t, d, ts, y, st, cont=True)
                    if S.cells_started(ode) >= n:
                        break
                S.set_yield(ode, None)
            torch.cuda.synchronize()
            got.append([a.cpu().numpy() for a in (y, t, d, st)])
        finally:
            S.CloseOdevec(ode)
    _same(got[1], got[0])
    assert np.all(got[0][3] == (4 if max_attempts else 0))


@pytest.mark.parametrize("cells", [(4096, 5000, 40), (33, 70, 700)])
def test_multi_block_jobs_fp32_factors(gpu_lib, cells):
    """FP32 factors in one launch whose blocks go from one job's kernel to
    another's: the bits of separate solves."""
    import torch
    from odevec_b200.multi import SolveMany
    S = gpu_lib
    got = []
    for fused in (True, False):
        wls = [W.rober(cells[0], seed=2), W.primordial(cells[1], seed=2), W.syn64(cells[2], seed=2)]
        wls[2].t_stop[:] = 1e2
        odes, jobs = [], []
        for wl in wls:
            odes.append(_solver(S, wl, nvector=1, precision="fp32_lu", escalation=False))
            jobs.append((odes[-1], *[torch.tensor(a, device="cuda") for a in (wl.t0, wl.dt0, wl.t_stop, wl.y)]))
        try:
            if fused:
                SolveMany(jobs, fused=True).run()
            else:
                for ode, t, d, ts, y in jobs:
                    S.SolveODE(ode, t, d, ts, y)
            torch.cuda.synchronize()
            got.append([a.cpu().numpy() for ode, t, d, ts, y in jobs for a in (y, t, d, ode.status)])
        finally:
            for ode in odes:
                S.CloseOdevec(ode)
    for a, b in zip(*got):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("precision,cells", [("fp64", 700), ("fp64", 151552), ("fp64", 151553), ("fp32_lu", 56833)])
def test_resumed_on_chip(gpu_lib, precision, cells):
    """A solve and its continuation at the sizes where either leaves the shape
    with the factors on chip: state and statistics as in a shape
    that the caller fixes."""
    import torch
    S = gpu_lib
    wl = W.primordial(ncells=cells, seed=6)
    wl.t_stop[:] = 1e6
    got = []
    for kw in ({}, {"staging": 9, "grid_blocks": 148}):
        ode = _solver(S, wl, precision=precision, escalation=False, **kw)
        try:
            y, t, d = (torch.tensor(a, device="cuda") for a in (wl.y, wl.t0, wl.dt0))
            ws = S.Workspace(ode, cells)
            for k in (1, 2):
                t, d = S.SolveODE(ode, t, d, torch.tensor(wl.t_stop * k, device="cuda"), y, workspace=ws,
                                  resume=k > 1)
            torch.cuda.synchronize()
            got.append([a.cpu().numpy() for a in (y, t, d, ode.status, ode.stats)])
        finally:
            S.CloseOdevec(ode)
    _same(got[0], got[1])


@pytest.mark.parametrize("na,nb", [(20000, 30000), (20000, 40000), (80000, 5000)])
def test_continuation_of_a_replayed_solve(gpu_lib, oracle, na, nb):
    """A captured solve yields and is continued after another solve on the same
    solver, whose rate table is a larger one, or which has a visit order where
    the captured one has none, or the other way round: the continuation takes
    the rates and the order of its own cells."""
    import torch
    S = gpu_lib
    a, b = W.primordial(ncells=na, seed=31), W.primordial(ncells=nb, seed=32)
    for wl in (a, b):
        wl.t_stop[:] = 1e6
    ode = _solver(S, a)
    try:
        flag = torch.zeros(1, dtype=torch.int32, device="cuda")
        S.set_yield(ode, flag)
        y, t, d, ts = (torch.tensor(v, device="cuda") for v in (a.y, a.t0, a.dt0, a.t_stop))
        init = [v.clone() for v in (y, t, d)]
        st = torch.zeros(a.ncells, dtype=torch.int32, device="cuda")
        S.SolveODERange(ode, 0, a.ncells, t, d, ts, y, st) # sizes the table
        torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            S.SolveODERange(ode, 0, a.ncells, t, d, ts, y, st)
        _same(_gpu(S, ode, b), _oracle(oracle, b))
        for v, v0 in zip((y, t, d), init):
            v.copy_(v0)
        flag.fill_(1)
        g.replay()
        assert S.cells_started(ode) < a.ncells
        flag.zero_()
        S.SolveODERange(ode, 0, a.ncells, t, d, ts, y, st, cont=True)
        torch.cuda.synchronize()
        _same([v.cpu().numpy() for v in (y, t, d, st)], _oracle(oracle, a)[:4])
        S.set_yield(ode, None)
    finally:
        S.CloseOdevec(ode)


def test_solve_beside_a_capture(gpu_lib, oracle):
    """A solve on one stream, which allocates its rate table, while another
    stream is being captured in the global mode: both come out whole."""
    import torch
    S = gpu_lib
    wl = W.primordial(ncells=5000, seed=33)
    wl.t_stop[:] = 1e6
    ode = _solver(S, wl)
    try:
        y, t, d, ts = (torch.tensor(v, device="cuda") for v in (wl.y, wl.t0, wl.dt0, wl.t_stop))
        st = torch.zeros(wl.ncells, dtype=torch.int32, device="cuda")
        x = torch.ones(64, device="cuda")
        other = torch.cuda.Stream()
        torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            x.add_(1.0)
            S.SolveODERange(ode, 0, wl.ncells, t, d, ts, y, st, stream=other)
        g.replay()
        torch.cuda.synchronize()
        assert float(x[0]) == 2.0
        _same([v.cpu().numpy() for v in (y, t, d, st)], _oracle(oracle, wl)[:4])
    finally:
        S.CloseOdevec(ode)


def test_multi_jobs_of_one_network(gpu_lib):
    """Two jobs of one network in one launch keep the bits of one job of all the
    cells, and its time: a warp that has left the first job's loop must not
    take the lockstep words from those that have not (each of their trips then
    waits out its limit, ten times the time)."""
    import torch
    from odevec_b200.multi import SolveMany
    S = gpu_lib
    n = 60000
    wl = W.primordial(ncells=n, seed=14)
    got, ms = [], []
    for cut in (n, n // 2):
        odes = [_solver(S, wl) for _ in range(n // cut)]
        try:
            best = None
            for _ in range(3):
                jobs = []
                for k, ode in enumerate(odes):
                    part = slice(k * cut, (k + 1) * cut)
                    jobs.append((ode, *[torch.tensor(a[..., part], device="cuda")
                                        for a in (wl.t0, wl.dt0, wl.t_stop, wl.y)]))
                many = SolveMany(jobs, fused=True)
                e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
                torch.cuda.synchronize()
                e0.record()
                many.run()
                e1.record()
                torch.cuda.synchronize()
                best = e0.elapsed_time(e1) if best is None else min(best, e0.elapsed_time(e1))
            got.append([torch.cat([j[k] for j in jobs], dim=-1).cpu().numpy() for k in (1, 2, 4)])
            ms.append(best)
        finally:
            for ode in odes:
                S.CloseOdevec(ode)
    for a, b in zip(*got):
        assert np.array_equal(a, b)
    assert ms[1] < 3.0 * ms[0], ms


@pytest.mark.parametrize("n", [75775, 75776])
def test_multi_block_limit(gpu_lib, n):
    """The large network's cells in a launch of several networks, in FP64 below
    and from the line on where they run one to a thread: the bits of separate
    solves."""
    import torch
    from odevec_b200.multi import SolveMany
    S = gpu_lib
    got = []
    for fused in (True, False):
        wls = [W.rober(33, seed=2), W.syn64(n, seed=12), W.primordial(5000, seed=2)]
        wls[1].t_stop[:] = 1e-6
        odes, jobs = [], []
        for wl in wls:
            odes.append(_solver(S, wl, nvector=1))
            jobs.append((odes[-1], *[torch.tensor(a, device="cuda") for a in (wl.t0, wl.dt0, wl.t_stop, wl.y)]))
        try:
            if fused:
                SolveMany(jobs, fused=True).run()
            else:
                for ode, t, d, ts, y in jobs:
                    S.SolveODE(ode, t, d, ts, y)
            torch.cuda.synchronize()
            got.append([a.cpu().numpy() for ode, t, d, ts, y in jobs for a in (y, t, d, ode.status)])
        finally:
            for ode in odes:
                S.CloseOdevec(ode)
    for a, b in zip(*got):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("precision", ["fp64_fma", "fp32_lu"])
def test_block_kernel_forms_masked_and_resumed(gpu_lib, precision):
    """The contracted forms with masked cells and CheckNegatives, then resumed:
    the bits of a thread per cell (staging 15)."""
    import torch
    S = gpu_lib
    wl = W.syn64(ncells=300, seed=15)
    wl.t_stop[:] = 10.0 ** np.random.default_rng(3).uniform(-3.0, 3.0, 300)
    mask = np.random.default_rng(4).random(300) > 0.2
    got = []
    for staging in (18, 15):
        ode = _solver(S, wl, precision=precision, staging=staging, escalation=False, CheckNegatives=True)
        try:
            y, t, d = (torch.tensor(a, device="cuda") for a in (wl.y, wl.t0, wl.dt0))
            ws = S.Workspace(ode, wl.ncells)
            for k, resume in enumerate((False, True, "en_old")):
                t, d = S.SolveODE(ode, t, d, torch.tensor(wl.t_stop * 2.0 ** k, device="cuda"), y, Mask=mask,
                                  workspace=ws, resume=resume)
            torch.cuda.synchronize()
            got.append([a.cpu().numpy() for a in (y, t, d, ode.status, ode.stats)])
        finally:
            S.CloseOdevec(ode)
    _same(got[0], got[1])


def test_block_kernel_visit_order(gpu_lib):
    """Cells of a large network visited longest span first, and in the given
    order as ranges below the size from which there is an order: the same
    bits."""
    import torch
    S = gpu_lib
    n = 40000
    wl = W.syn64(ncells=n, seed=16)
    wl.t_stop[:] = 10.0 ** np.random.default_rng(5).uniform(-6.0, 0.0, n)
    got = []
    for ranges in ([(0, n)], [(0, 25000), (25000, n)]):
        ode = _solver(S, wl)
        try:
            y, t, d, ts = (torch.tensor(a, device="cuda") for a in (wl.y, wl.t0, wl.dt0, wl.t_stop))
            st = torch.zeros(n, dtype=torch.int32, device="cuda")
            for c0, c1 in ranges:
                S.SolveODERange(ode, c0, c1, t, d, ts, y, st)
            torch.cuda.synchronize()
            got.append([a.cpu().numpy() for a in (y, t, d, st)])
        finally:
            S.CloseOdevec(ode)
    _same(got[0], got[1])


def test_captured_solve_beyond_its_table(gpu_lib, oracle):
    """A captured solve of more cells than the solver's rate table holds: the
    solve kernel evaluates the rates."""
    import torch
    S = gpu_lib
    a, b = W.primordial(ncells=4096, seed=34), W.primordial(ncells=9000, seed=35)
    for wl in (a, b):
        wl.t_stop[:] = 1e6
    ode = _solver(S, b)
    try:
        _gpu(S, ode, a)
        y, t, d, ts = (torch.tensor(v, device="cuda") for v in (b.y, b.t0, b.dt0, b.t_stop))
        st = torch.zeros(b.ncells, dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            S.SolveODERange(ode, 0, b.ncells, t, d, ts, y, st)
        g.replay()
        torch.cuda.synchronize()
        _same([v.cpu().numpy() for v in (y, t, d, st)], _oracle(oracle, b)[:4])
    finally:
        S.CloseOdevec(ode)


@pytest.mark.parametrize("group", [1, 32])
def test_step_choice_ties(gpu_lib, oracle, group):
    """Cells at rest, whose corrections are zero, so that all candidates of the
    step-size choice are equal, beside ordinary ones."""
    wl = W.rober(ncells=96, seed=17)
    wl.y[:, 32:64] = np.array([0.0, 0.0, 1.0])[:, None]
    ode = _solver(gpu_lib, wl, nvector=group)
    try:
        _same(_gpu(gpu_lib, ode, wl), _oracle(oracle, wl, group=group))
    finally:
        gpu_lib.CloseOdevec(ode)

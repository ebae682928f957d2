"""Resolved task graphs executed by the device scheduler in its three forms (persistent
kernel, one launch per task, CUDA graph): results bit-exact against the oracle."""
import numpy as np
import pytest

import kernels_oracle as O
import streams as S
import xkaapi_b200 as xk

pytestmark = pytest.mark.gpu
C = 0.2


class _DevView:
    def __init__(self, ptr, n, typestr="<i4"):
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": typestr, "data": (ptr, False), "version": 3}


def heat_graph(torch, nx, ny, ts, steps, f32=False, seed=42):
    dt = np.float32 if f32 else np.float64
    g = O.heat_init(nx, ny, seed=seed).astype(dt)
    a = torch.from_numpy(g).cuda(); b = torch.from_numpy(g).cuda()
    esz = 4 if f32 else 8
    recs = S.heat_stream(nx, ny, ts, ts, steps, base_src=a.data_ptr(), base_dst=b.data_ptr(), s=esz)
    res = xk.Resolver()
    res.add(recs)
    descs = xk.heat_task_descs((a.data_ptr(), b.data_ptr()), nx, ny, nx, ts, ts, steps, C, f32=f32)
    return g, a, b, res, descs


@pytest.mark.parametrize("form", [xk.FORM_PERSISTENT, xk.FORM_PLAIN, xk.FORM_GRAPH])
@pytest.mark.parametrize("nx,ny,ts,steps", [(1024, 1024, 128, 100), (300, 200, 64, 7)])
def test_heat_forms_bit_exact(torch_cuda, form, nx, ny, ts, steps):
    torch = torch_cuda
    if form == xk.FORM_GRAPH and steps > 20:
        steps = 20                           # keep graph instantiation short
    g, a, b, res, descs = heat_graph(torch, nx, ny, ts, steps)
    sch = xk.Scheduler()
    sch.set_tasks(descs)
    sch.run(res.graph(), form)
    n = sch.wait()
    if form == xk.FORM_PERSISTENT:
        assert n == len(descs)
    out = (a if steps % 2 == 0 else b).cpu().numpy()
    np.testing.assert_array_equal(out, O.heat_run(g, nx, ny, steps, C))
    sch.close(); res.close()


def test_heat_f32_persistent(torch_cuda):
    torch = torch_cuda
    nx = ny = 512
    g, a, b, res, descs = heat_graph(torch, nx, ny, 128, 30, f32=True)
    sch = xk.Scheduler(); sch.set_tasks(descs); sch.run(res.graph()); sch.wait()
    out = a.cpu().numpy()
    np.testing.assert_array_equal(out, O.heat_run(g, nx, ny, 30, C, dtype=np.float32))
    ref64 = O.heat_run(g.astype(np.float64), nx, ny, 30, C)
    assert np.abs(out.astype(np.float64) - ref64).max() / np.abs(ref64).max() <= 1e-5


def test_persistent_small_grid_many_ctas(torch_cuda):
    # more CTAs than ready tasks at any time: idle CTAs wait on queue slots and still finish
    torch = torch_cuda
    g, a, b, res, descs = heat_graph(torch, 256, 256, 64, 40)
    sch = xk.Scheduler(); sch.set_grid(600); sch.set_tasks(descs); sch.run(res.graph()); sch.wait()
    np.testing.assert_array_equal(a.cpu().numpy(), O.heat_run(g, 256, 256, 40, C))


def axpby_chain(torch, n, passes, seed):
    """y = a*x + b*y over seeded chunkings whose boundaries move between passes (segment
    accesses: R on the x chunk, RW on the y chunk)."""
    rng = np.random.default_rng(seed)
    x = rng.uniform(-1, 1, n); y = rng.uniform(-1, 1, n)
    dx, dy = torch.from_numpy(x).cuda(), torch.from_numpy(y).cuda()
    tasks, chunks = [], []
    for p in range(passes):
        a, b = rng.uniform(-2, 2, 2)
        off = int(rng.integers(1, 97))
        cuts = [0, off]
        while cuts[-1] < n:
            cuts.append(min(n, cuts[-1] + int(rng.integers(1, max(2, n // 6)))))
        for lo, hi in zip(cuts[:-1], cuts[1:]):
            if lo < hi:
                tasks.append([("s", S.R, dx.data_ptr() + 8 * lo, dx.data_ptr() + 8 * hi),
                              ("s", S.RW, dy.data_ptr() + 8 * lo, dy.data_ptr() + 8 * hi)])
                chunks.append((lo, hi, a, b))
    ref = y.copy()
    for lo, hi, a, b in chunks:
        ref[lo:hi] = O.axpby(a, x[lo:hi], b, ref[lo:hi])
    descs = np.zeros(len(chunks), dtype=xk.axpby_desc_dtype())
    descs["kind"] = xk.TASK_AXPBY; descs["x"] = dx.data_ptr(); descs["y"] = dy.data_ptr()
    descs["lo"] = [c[0] for c in chunks]; descs["hi"] = [c[1] for c in chunks]
    descs["a"] = [c[2] for c in chunks]; descs["b"] = [c[3] for c in chunks]
    return S.from_tuples(tasks), descs, dy, ref


@pytest.mark.parametrize("form", [xk.FORM_PERSISTENT, xk.FORM_PLAIN, xk.FORM_GRAPH])
def test_axpby_chains(torch_cuda, form):
    torch = torch_cuda
    recs, descs, dy, ref = axpby_chain(torch, 200_003, 10, 7)
    res = xk.Resolver(); res.add(recs)
    sch = xk.Scheduler(); sch.set_tasks(descs); sch.run(res.graph(), form); sch.wait()
    np.testing.assert_array_equal(dy.cpu().numpy(), ref)


def test_timeout_returns_error_and_context_survives(torch_cuda):
    """A task whose wait counter never reaches zero: the persistent CTAs give up after the
    time limit, the kernel returns, xkb_sched_wait reports XKB_ETIMEDOUT; the context is
    then reused for a valid graph."""
    torch = torch_cuda
    ptr = torch.zeros(3, dtype=torch.int32, device="cuda")          # no edges
    succ = torch.zeros(1, dtype=torch.int32, device="cuda")
    npred = torch.tensor([0, 1], dtype=torch.int32, device="cuda")   # task 1 waits for nobody's release
    g = xk.TaskGraph(2, 0, ptr.data_ptr(), succ.data_ptr(), npred.data_ptr())
    descs = np.zeros(2, dtype=xk.task_desc_dtype())                 # two no-op tasks
    sch = xk.Scheduler(); sch.set_tasks(descs); sch.set_timeout(0.2); sch.set_grid(4)
    sch.run(g)
    with pytest.raises(xk.XkbError) as e:
        sch.wait()
    assert e.value.code == xk.XKB_ETIMEDOUT
    g2, a, b, res, d2 = heat_graph(torch, 128, 128, 64, 4)
    sch.set_tasks(d2); sch.run(res.graph()); sch.wait()
    np.testing.assert_array_equal(a.cpu().numpy(), O.heat_run(g2, 128, 128, 4, C))


@pytest.mark.parametrize("team", [1, 2, 4, 8])
def test_heat_persistent_team_sizes(torch_cuda, team):
    torch = torch_cuda
    g, a, b, res, descs = heat_graph(torch, 300, 200, 64, 9)
    sch = xk.Scheduler(); sch.set_team(team); sch.set_tasks(descs); sch.run(res.graph())
    assert sch.wait() == len(descs)
    np.testing.assert_array_equal(b.cpu().numpy(), O.heat_run(g, 300, 200, 9, C))


@pytest.mark.parametrize("team", [1, 8])
def test_axpby_chains_team_sizes(torch_cuda, team):
    torch = torch_cuda
    recs, descs, dy, ref = axpby_chain(torch, 50_001, 6, 3)
    res = xk.Resolver(); res.add(recs)
    sch = xk.Scheduler(); sch.set_team(team); sch.set_tasks(descs); sch.run(res.graph()); sch.wait()
    np.testing.assert_array_equal(dy.cpu().numpy(), ref)


@pytest.mark.parametrize("steps", [1, 2, 7, 10])
def test_periodic_heat_one_launch(torch_cuda, steps):
    """Three resolved two-step windows -> periodic form; one persistent launch runs all steps
    (a half window at the end for odd step counts) and gives the oracle's grid."""
    torch = torch_cuda
    nx, ny, ts = 300, 200, 64
    g0 = O.heat_init(nx, ny, seed=21)
    a = torch.from_numpy(g0).cuda(); b = torch.from_numpy(g0).cuda()
    res = xk.Resolver()
    res.add(xk.heat_access_records(nx, ny, ts, ts, 0, 6, a.data_ptr(), b.data_ptr()))
    per_step = (-(-nx // ts)) * (-(-ny // ts))
    pg = res.periodic(2 * per_step)
    sch = xk.Scheduler()
    sch.set_tasks(xk.heat_task_descs((a.data_ptr(), b.data_ptr()), nx, ny, nx, ts, ts, 2, C))
    sch.run_periodic(pg, (steps + 1) // 2, per_step if steps % 2 else 2 * per_step)
    assert sch.wait() == steps * per_step
    out = (a if steps % 2 == 0 else b).cpu().numpy()
    np.testing.assert_array_equal(out, O.heat_run(g0, nx, ny, steps, C))


def test_periodic_rejects_aperiodic_graph(torch_cuda):
    recs = S.microbench_stream(30, 1, n=512, ld=512)
    res = xk.Resolver(); res.add(recs)
    with pytest.raises(xk.XkbError):
        res.periodic(10)


@pytest.mark.parametrize("nx,ny,ts,steps,f32,team", [
    (1024, 768, 128, 12, False, 2), (300, 200, 64, 9, False, 1), (300, 200, 100, 9, False, 8),
    (301, 203, 64, 6, False, 2),                       # rows not 16-byte aligned: register body
    (516, 260, 128, 10, True, 2), (514, 130, 64, 6, True, 4), (1000, 1000, 96, 8, True, 1)])
def test_bulk_staged_body_matches_register_body(torch_cuda, nx, ny, ts, steps, f32, team):
    """The bulk-staged tile body (default) and the register body give the oracle's grid bit for
    bit, for FP64 and FP32 storage, tiles that are not a multiple of the strip, and grids whose
    rows cannot be staged (odd FP64 / non-multiple-of-4 FP32 widths fall back)."""
    torch = torch_cuda
    dt = np.float32 if f32 else np.float64
    want = O.heat_run(O.heat_init(nx, ny, seed=5), nx, ny, steps, C, dtype=dt)
    for bulk in (True, False):
        g, a, b, res, descs = heat_graph(torch, nx, ny, ts, steps, f32=f32, seed=5)
        sch = xk.Scheduler(); sch.set_team(team); sch.set_staging(bulk); sch.set_tasks(descs)
        sch.run(res.graph())
        assert sch.wait() == len(descs)
        np.testing.assert_array_equal((a if steps % 2 == 0 else b).cpu().numpy(), want)
        sch.close(); res.close()


@pytest.mark.parametrize("nx,ny,ts,steps,f32", [
    (130, 70, 128, 7, False),       # 2 tiles (one a sliver): 32 units each, some without a column
    (200, 136, 64, 9, True),        # 12 tiles: 32 units, several CTAs per tile
    (1024, 640, 64, 5, False),      # 160 tiles: 8 units, one CTA per tile
    (1152, 1152, 48, 4, True),      # 576 tiles: 8 units, warps take them one by one
    (1700, 1500, 48, 3, False),     # 1152 tiles: 4 units
    (3000, 3000, 48, 3, False)])    # 3969 tiles: not split
@pytest.mark.parametrize("order", ["in order", "queue", "periodic"])
def test_heat_units_and_orders(torch_cuda, nx, ny, ts, steps, f32, order):
    """Every split of a tile task into units, taken in spawn order, through the ready queue (two
    graphs spawned one after the other are not spawned level by level), and in order over the
    windows of a periodic graph with a partial last window: the oracle's grids bit for bit."""
    torch = torch_cuda
    dt = np.float32 if f32 else np.float64
    per_step = (-(-nx // ts)) * (-(-ny // ts))
    graphs = 2 if order == "queue" else 1
    window = 2 if order == "periodic" else steps
    grids, recs, descs = [], [], []
    for k in range(graphs):
        g = O.heat_init(nx, ny, seed=60 + k).astype(dt)
        a, b = torch.from_numpy(g).cuda(), torch.from_numpy(g).cuda()
        r = xk.heat_access_records(nx, ny, ts, ts, 0, 6 if order == "periodic" else steps, a.data_ptr(), b.data_ptr(), esize=dt().itemsize)
        r["task"] += k * steps * per_step
        grids.append((g, a, b)); recs.append(r)
        descs.append(xk.heat_task_descs((a.data_ptr(), b.data_ptr()), nx, ny, nx, ts, ts, window, C, f32=f32))
    res = xk.Resolver(); res.add(np.concatenate(recs))
    sch = xk.Scheduler(); sch.set_tasks(np.concatenate(descs))
    if order == "periodic":
        sch.run_periodic(res.periodic(2 * per_step), (steps + 1) // 2, per_step if steps % 2 else 2 * per_step)
    else:
        sch.run(res.graph())
    assert sch.wait() == graphs * steps * per_step
    for g, a, b in grids:
        np.testing.assert_array_equal((a if steps % 2 == 0 else b).cpu().numpy(), O.heat_run(g, nx, ny, steps, C, dtype=dt))
    sch.close(); res.close()


@pytest.mark.parametrize("lo", [0, 1])
@pytest.mark.parametrize("n", [1, 2, 255, 256, 8191, 8192, 8193, 3 * 8192 + 5, 300_001])
def test_axpby_units(torch_cuda, n, lo):
    """One axpby task over n elements from an aligned and an unaligned start, split into pieces of
    8192 elements: every element updated once, nothing outside the range touched."""
    torch = torch_cuda
    rng = np.random.default_rng(n)
    x, y = rng.uniform(-1, 1, n + 4), rng.uniform(-1, 1, n + 4)
    dx, dy = torch.from_numpy(x).cuda(), torch.from_numpy(y).cuda()
    d = np.zeros(1, dtype=xk.axpby_desc_dtype())
    d["kind"], d["x"], d["y"], d["lo"], d["hi"], d["a"], d["b"] = xk.TASK_AXPBY, dx.data_ptr(), dy.data_ptr(), lo, lo + n, 0.3, -1.7
    res = xk.Resolver()
    res.add(S.from_tuples([[("s", S.RW, dy.data_ptr() + 8 * lo, dy.data_ptr() + 8 * (lo + n))]]))
    sch = xk.Scheduler(); sch.set_tasks(d); sch.run(res.graph())
    assert sch.wait() == 1
    y[lo:lo + n] = O.axpby(0.3, x[lo:lo + n], -1.7, y[lo:lo + n])
    np.testing.assert_array_equal(dy.cpu().numpy(), y)


@pytest.mark.parametrize("f32", [False, True])
@pytest.mark.parametrize("nx,ny,ld,ts,steps", [(131, 77, 131, 40, 5), (260, 150, 261, 64, 5), (1027, 300, 1027, 64, 4),
                                               (130, 90, 132, 32, 5), (2310, 2500, 2310, 48, 3)])
def test_heat_grids_of_any_alignment(torch_cuda, nx, ny, ld, ts, steps, f32):
    """Graphs on grids with odd leading dimensions (the row-by-row kernels), with a last vector past
    the last row, and one wide enough to take its tiles column by column: bit-exact, padding intact."""
    torch = torch_cuda
    dt = np.float32 if f32 else np.float64
    g = np.full((ny, ld), 7.0, dtype=dt)
    g[:, :nx] = O.heat_init(nx, ny, seed=nx).astype(dt)
    a, b = torch.from_numpy(g).cuda(), torch.from_numpy(g).cuda()
    res = xk.Resolver()
    res.add(xk.heat_access_records(nx, ny, ts, ts, 0, steps, a.data_ptr(), b.data_ptr(), esize=dt().itemsize, ld=ld))
    sch = xk.Scheduler()
    sch.set_tasks(xk.heat_task_descs((a.data_ptr(), b.data_ptr()), nx, ny, ld, ts, ts, steps, C, f32=f32))
    sch.run(res.graph())
    sch.wait()
    out = (a if steps % 2 == 0 else b).cpu().numpy()
    want = O.heat_run(np.ascontiguousarray(g[:, :nx]), nx, ny, steps, C, dtype=dt)
    np.testing.assert_array_equal(out[:, :nx], want.reshape(ny, nx))
    assert (out[:, nx:] == 7.0).all()
    sch.close(); res.close()


@pytest.mark.parametrize("fan", [3, 40, 100])
def test_split_task_releases_successors_behind_all_its_units(torch_cuda, fan):
    """Queue runs of split tasks with more successors than one lane, or one warp, decrements: a
    producer of 64 pieces, `fan` consumers that wait for all of it, a producer that waits for theirs,
    and so on. Two such graphs one after the other are not spawned level by level, so they take the queue."""
    torch = torch_cuda
    n, levels = 64 * 8192, 6
    rng = np.random.default_rng(fan)
    cuts = np.linspace(0, n, fan + 1).astype(np.int64)
    tasks, descs, checks = [], [], []
    for _ in range(2):
        y, z = rng.uniform(-1, 1, n), rng.uniform(-1, 1, n)
        dy, dz = torch.from_numpy(y).cuda(), torch.from_numpy(z).cuda()
        for level in range(levels):
            a, b = rng.uniform(-1, 1, 2)
            whole = level % 2 == 0
            src, dst, hs, hd = (dz, dy, z, y) if whole else (dy, dz, y, z)
            for lo, hi in [(0, n)] if whole else zip(cuts[:-1], cuts[1:]):
                tasks.append([("s", S.R, src.data_ptr(), src.data_ptr() + 8 * n),
                              ("s", S.RW, dst.data_ptr() + 8 * int(lo), dst.data_ptr() + 8 * int(hi))])
                descs.append((src.data_ptr(), dst.data_ptr(), int(lo), int(hi), a, b))
                hd[lo:hi] = O.axpby(a, hs[lo:hi], b, hd[lo:hi])
        checks += [(dy, y), (dz, z)]
    d = np.zeros(len(descs), dtype=xk.axpby_desc_dtype())
    d["kind"] = xk.TASK_AXPBY
    for k, f in enumerate(("x", "y", "lo", "hi", "a", "b")):
        d[f] = [t[k] for t in descs]
    res = xk.Resolver(); res.add(S.from_tuples(tasks))
    sch = xk.Scheduler(); sch.set_tasks(d); sch.run(res.graph())
    assert sch.wait() == len(d)
    for got, want in checks:
        np.testing.assert_array_equal(got.cpu().numpy(), want)
    sch.close(); res.close()


def chains(torch, count, length, roots):
    """`roots` heat tiles, then `count` chains of `length` tiles, spawned chain by chain; every chain
    follows one of the roots, if there are any. Returns the graph, the descriptors, what keeps them
    alive, and each chain's grids with the seed of its initial one."""
    side, grids, descs, edges = 128, [], [], []
    for k in range(roots + count):
        g = O.heat_init(side, side, seed=k)
        a, b = torch.from_numpy(g).cuda(), torch.from_numpy(g).cuda()
        grids.append((k, a, b))
        descs.append(xk.heat_task_descs((a.data_ptr(), b.data_ptr()), side, side, side, side, side, 1 if k < roots else length, C))
        if k >= roots:
            first = roots + (k - roots) * length
            edges += [(first + i, first + i + 1) for i in range(length - 1)]
            if roots:
                edges.append((k % roots, first))
    descs = np.concatenate(descs)
    edges = np.array(sorted(edges), dtype=np.int64)
    ptr = np.concatenate([[0], np.cumsum(np.bincount(edges[:, 0], minlength=len(descs)))])
    keep = [torch.from_numpy(v.astype(np.int32)).cuda() for v in (ptr, edges[:, 1], np.bincount(edges[:, 1], minlength=len(descs)))]
    return xk.TaskGraph(len(descs), len(edges), *(v.data_ptr() for v in keep)), descs, keep, grids[roots:]


@pytest.mark.parametrize("roots", [1, 2])
def test_chains_behind_common_roots_run_side_by_side(torch_cuda, roots):
    """Chains spawned one after the other behind a first task or two that all of them follow: taken in
    spawn order they would run one after another. They take about as long as without the roots (a
    small part of what one after another takes), and every grid is the oracle's."""
    torch = torch_cuda
    ms = {}
    for r in (0, roots):
        graph, descs, keep, grids = chains(torch, 64, 100, r)
        sch = xk.Scheduler(); sch.set_tasks(descs)
        sch.run(graph)
        assert sch.wait() == len(descs)
        for seed, a, b in grids:
            np.testing.assert_array_equal(a.cpu().numpy(), O.heat_run(O.heat_init(128, 128, seed=seed), 128, 128, 100, C))
        ms[r] = []
        for _ in range(5):
            sch.run(graph); sch.wait()
            ms[r].append(sch.kernel_ms())
        sch.close()
    assert min(ms[roots]) < 2 * min(ms[0]), ms


def one_axpby_task(torch, n):
    x, y = torch.rand(n, dtype=torch.float64, device="cuda"), torch.rand(n, dtype=torch.float64, device="cuda")
    d = np.zeros(1, dtype=xk.axpby_desc_dtype())
    d["kind"], d["x"], d["y"], d["hi"], d["a"], d["b"] = xk.TASK_AXPBY, x.data_ptr(), y.data_ptr(), n, 0.5, 0.25
    keep = [torch.zeros(k, dtype=torch.int32, device="cuda") for k in (2, 1, 1)]
    return xk.TaskGraph(1, 0, *(v.data_ptr() for v in keep)), d, [x, y, keep]


def best_ms(sch, graph, reps=5):
    sch.run(graph); sch.wait()
    ms = []
    for _ in range(reps):
        sch.run(graph); sch.wait()
        ms.append(sch.kernel_ms())
    return min(ms)


def test_team_is_what_the_caller_sets(torch_cuda):
    """A caller that sets the warps per task gets that many: an axpby task of 512 pieces takes one warp
    several times as long as eight, and these several times as long as the split that the
    scheduler chooses by itself (256 warps)."""
    torch = torch_cuda
    graph, d, keep = one_axpby_task(torch, 512 * 8192)
    ms = {}
    for team in (None, 8, 1):
        sch = xk.Scheduler(); sch.set_tasks(d)
        if team:
            sch.set_team(team)
        ms[team] = best_ms(sch, graph)
        sch.close()
    assert ms[1] > 3 * ms[8] and ms[8] > 3 * ms[None], ms


@pytest.mark.parametrize("first", ["long axpby", "heat tile"])
def test_split_fits_the_tasks_behind_the_first(torch_cuda, first):
    """The one task that is ready at the start does not choose the split for what follows: a long axpby
    task before 60,000 short ones, and a single tile before 4,096 tiles a step. The automatic split is
    not slower than one warp per task (to a margin of a half), and the results are the oracle's."""
    torch = torch_cuda
    rng = np.random.default_rng(4)
    if first == "long axpby":
        n, short, m = 64 * 8192, 60_000, 64
        host = [rng.uniform(-1, 1, n), rng.uniform(-1, 1, n), rng.uniform(-1, 1, short * m), rng.uniform(-1, 1, short * m)]
        x, y, u, v = dev = [torch.from_numpy(h).cuda() for h in host]
        d = np.zeros(1 + short, dtype=xk.axpby_desc_dtype())
        d["kind"], d["a"], d["b"] = xk.TASK_AXPBY, 0.5, 0.25
        d["x"], d["y"], d["lo"] = u.data_ptr(), v.data_ptr(), (np.arange(1 + short) - 1) * m
        d["hi"] = d["lo"] + m
        d["x"][0], d["y"][0], d["lo"][0], d["hi"][0] = x.data_ptr(), y.data_ptr(), 0, n
        edges = np.stack([np.zeros(short, np.int64), 1 + np.arange(short)], axis=1)
    else:
        side, ts, steps = 2048, 32, 6
        g = O.heat_init(side, side, seed=8)
        small = O.heat_init(64, 64, seed=9)
        a, b, p, q = dev = [torch.from_numpy(h).cuda() for h in (g, g, small, small)]
        d = np.concatenate([xk.heat_task_descs((p.data_ptr(), q.data_ptr()), 64, 64, 64, 64, 64, 1, C),
                            xk.heat_task_descs((a.data_ptr(), b.data_ptr()), side, side, side, ts, ts, steps, C)])
        per = (side // ts) ** 2
        r = xk.Resolver()
        r.add(xk.heat_access_records(side, side, ts, ts, 0, steps, a.data_ptr(), b.data_ptr()))
        e = r.edges().astype(np.int64)
        r.close()
        edges = np.concatenate([np.stack([np.zeros(per, np.int64), 1 + np.arange(per)], axis=1), e + 1])
    edges = edges[np.lexsort((edges[:, 1], edges[:, 0]))]
    ptr = np.concatenate([[0], np.cumsum(np.bincount(edges[:, 0], minlength=len(d)))])
    keep = [torch.from_numpy(w.astype(np.int32)).cuda() for w in (ptr, edges[:, 1], np.bincount(edges[:, 1], minlength=len(d)))]
    graph = xk.TaskGraph(len(d), len(edges), *(w.data_ptr() for w in keep))
    sch = xk.Scheduler(); sch.set_tasks(d); sch.run(graph)
    assert sch.wait() == len(d)
    if first == "long axpby":
        np.testing.assert_array_equal(y.cpu().numpy(), O.axpby(0.5, host[0], 0.25, host[1]))
        np.testing.assert_array_equal(v.cpu().numpy(), O.axpby(0.5, host[2], 0.25, host[3]))
    else:
        np.testing.assert_array_equal(a.cpu().numpy(), O.heat_run(g, side, side, steps, C))
    auto = best_ms(sch, graph)
    sch.set_team(1)
    one = best_ms(sch, graph)
    sch.close()
    assert auto < 1.5 * one, (auto, one)


@pytest.mark.parametrize("group", [20, 33, 70, 200])
def test_many_successors_in_this_window_and_the_next(torch_cuda, group):
    """A periodic graph whose hub task has `group` successors in its own window and as many in the
    next one (its first `group` tasks), over a partial last window: the oracle's vectors."""
    torch = torch_cuda
    rng = np.random.default_rng(group)
    m, windows, tail = 40, 7, group + 1
    n = group * m
    y, z, u, v = (rng.uniform(-1, 1, n) for _ in range(4))
    dy, dz, du, dv = (torch.from_numpy(h).cuda() for h in (y, z, u, v))
    # u += y by slices, the hub y += z, v += y by slices
    window = [(dy, du, k * m, (k + 1) * m, 0.5, 0.75) for k in range(group)] + [(dz, dy, 0, n, -0.5, 0.75)] + \
             [(dy, dv, k * m, (k + 1) * m, 0.25, -0.75) for k in range(group)]
    d = np.zeros(len(window), dtype=xk.axpby_desc_dtype())
    d["kind"] = xk.TASK_AXPBY
    tasks = []
    for i, (src, dst, lo, hi, a, b) in enumerate(window):
        for name, val in (("x", src.data_ptr()), ("y", dst.data_ptr()), ("lo", lo), ("hi", hi), ("a", a), ("b", b)):
            d[name][i] = val
        tasks.append([("s", S.R, src.data_ptr() + 8 * lo, src.data_ptr() + 8 * hi), ("s", S.RW, dst.data_ptr() + 8 * lo, dst.data_ptr() + 8 * hi)])
    res = xk.Resolver(); res.add(S.from_tuples(tasks * 3))
    sch = xk.Scheduler(); sch.set_tasks(d)
    sch.run_periodic(res.periodic(len(window)), windows, tail)
    assert sch.wait() == (windows - 1) * len(window) + tail
    for w in range(windows):
        u = O.axpby(0.5, y, 0.75, u)
        y = O.axpby(-0.5, z, 0.75, y)
        if w + 1 < windows:
            v = O.axpby(0.25, y, -0.75, v)
    for got, want in ((du, u), (dy, y), (dv, v)):
        np.testing.assert_array_equal(got.cpu().numpy(), want)
    sch.close(); res.close()


def test_many_successors_of_one_task(torch_cuda):
    """60,000 tasks behind one, from the launch to the end: no step of it takes them one after the
    other. (One thread that looks through them takes 4 ms; the limit is what the run took when every
    graph went through the queue, 3.2 ms.)"""
    torch = torch_cuda
    n = 60_000
    ptr = torch.full((n + 2,), n, dtype=torch.int32, device="cuda"); ptr[0] = 0
    succ = 1 + torch.arange(n, dtype=torch.int32, device="cuda")
    npred = torch.ones(n + 1, dtype=torch.int32, device="cuda"); npred[0] = 0
    graph = xk.TaskGraph(n + 1, n, ptr.data_ptr(), succ.data_ptr(), npred.data_ptr())
    sch = xk.Scheduler(); sch.set_tasks(np.zeros(n + 1, dtype=xk.task_desc_dtype()))
    ms = []
    with torch.cuda.stream(torch.cuda.default_stream()):
        for _ in range(6):
            e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
            e[0].record(); sch.run(graph); e[1].record()
            assert sch.wait() == n + 1
            ms.append(e[0].elapsed_time(e[1]))
    sch.close()
    assert min(ms[1:]) < 3.2, ms


@pytest.mark.parametrize("skip", [0, 20, 61])
def test_graphs_that_begin_inside_a_step_run_in_order(torch_cuda, skip):
    """A heat graph without its first tasks, as a runtime hands it over in windows: where its first tasks are
    the ones ready at the start (some of the second step's last tiles are too when the first step is nearly
    done) it is taken in spawn order like the whole graph, about twice as fast as the queue (11 against 5
    us a step), and it ends with the oracle's grids."""
    torch = torch_cuda
    n, ts, steps = 1024, 128, 60
    g = O.heat_init(n, n, seed=3)
    after = O.heat_run(g, n, n, 1, C)
    r = xk.Resolver()
    r.add(xk.heat_access_records(n, n, ts, ts, 0, steps, 1 << 40, 1 << 41))
    e = r.edges().astype(np.int64)
    r.close()
    times = {}
    for extra in (0, 1):                       # a no-op task more, ready at the start behind all others: the queue
        a, b = torch.from_numpy(g).cuda(), torch.from_numpy(g).cuda()
        d = xk.heat_task_descs((a.data_ptr(), b.data_ptr()), n, n, n, ts, ts, steps, C)[skip:]
        d = np.concatenate([d, np.zeros(extra, dtype=d.dtype)])
        for t in range(skip):                  # the skipped tiles are there already
            x, y = t // 8 * ts, t % 8 * ts
            b[y:y + ts, x:x + ts] = torch.from_numpy(np.ascontiguousarray(after[y:y + ts, x:x + ts])).cuda()
        edges = e[(e >= skip).all(axis=1)] - skip
        edges = edges[np.lexsort((edges[:, 1], edges[:, 0]))]
        ptr = np.concatenate([[0], np.cumsum(np.bincount(edges[:, 0], minlength=len(d)))])
        npred = np.bincount(edges[:, 1], minlength=len(d))
        keep = [torch.from_numpy(w.astype(np.int32)).cuda() for w in (ptr, edges[:, 1], npred)]
        graph = xk.TaskGraph(len(d), len(edges), *(w.data_ptr() for w in keep))
        sch = xk.Scheduler(); sch.set_tasks(d); sch.run(graph)
        assert sch.wait() == len(d)
        np.testing.assert_array_equal(a.cpu().numpy(), O.heat_run(g, n, n, steps, C))
        if not extra:
            ready = np.flatnonzero(npred == 0)
            first = np.array_equal(ready, np.arange(len(ready)))
        times[extra] = best_ms(sch, graph)
        sch.close()
    assert first == (skip != 61)
    assert not first or times[0] < 0.75 * times[1], times


def test_units_of_the_longest_runs_are_numbered(torch_cuda):
    """A run of 2^29 tasks and eight warps per task would need more unit numbers than there are: tasks are
    split into fewer units there, whoever set their number, and every task runs once."""
    torch = torch_cuda
    period, windows = 1 << 16, (1 << 13) + 3
    ptr = torch.zeros(period + 1, dtype=torch.int32, device="cuda")
    each = torch.arange(period + 1, dtype=torch.int32, device="cuda")       # task t of a window follows task t of the one before
    none, one = torch.zeros(period, dtype=torch.int32, device="cuda"), torch.ones(period, dtype=torch.int32, device="cuda")
    graph = xk.PeriodicGraph(period, ptr.data_ptr(), none.data_ptr(), each.data_ptr(), each.data_ptr(), none.data_ptr(), one.data_ptr())
    sch = xk.Scheduler(); sch.set_team(8); sch.set_tasks(np.zeros(period, dtype=xk.task_desc_dtype()))
    sch.run_periodic(graph, windows)
    assert sch.wait() == period * windows
    sch.close()

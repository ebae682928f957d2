"""GPU dependency resolver: bit-exact unique edge sets against the reference's own trees
(golden fixtures) and against the oracle restatement on larger seeded streams."""
import os
import subprocess
import sys

import numpy as np
import pytest

import deps_util as U
import streams as S
import xkaapi_b200 as xk

pytestmark = pytest.mark.gpu
GOLDEN = np.load(U.os.path.join(U.REPO, "tests", "golden", "deps_golden.npz"))
CASES = sorted(k[:-len("__stream")] for k in GOLDEN.files if k.endswith("__stream"))


def gpu_edges(recs, batches=1, seed=0):
    r = xk.Resolver()
    for b in (U.split_batches(recs, batches, seed) if batches > 1 else [recs]):
        if len(b):
            r.add(b)
    e = r.edges()
    r.close()
    return e


def expanded(recs):
    """Concurrent-mode handle accesses go through the handle map's expansion first."""
    if not ((recs["reserved"] >> 8) == 4).any():
        return recs
    m = xk.HandleMap()
    out = m.expand(recs)
    m.close()
    return out


@pytest.mark.parametrize("case", CASES)
def test_golden_reference_edges(torch_cuda, case):
    np.testing.assert_array_equal(gpu_edges(expanded(GOLDEN[case + "__stream"])), GOLDEN[case + "__edges"])


@pytest.mark.parametrize("seed", range(3))
@pytest.mark.parametrize("batches", [1, 5])
def test_concurrent_handle_streams_vs_oracle(torch_cuda, seed, batches):
    """Longer concurrent-mode handle streams: the GPU resolver on the expanded stream (in batches)
    against the oracle's restatement of the handle map on the stream as spawned."""
    recs = S.handle_concurrent_stream(seed + 300, n=3000)
    np.testing.assert_array_equal(gpu_edges(expanded(recs), batches, seed=seed), U.oracle_edges(recs))


@pytest.mark.parametrize("case", ["heat_1024_t128_s3", "microbench_1024_2000", "mixed_segmat_0", "mixed_mat_1"])
@pytest.mark.parametrize("batches", [2, 7])
def test_incremental_batches_equal_one_shot(torch_cuda, case, batches):
    np.testing.assert_array_equal(gpu_edges(GOLDEN[case + "__stream"], batches, seed=batches),
                                  GOLDEN[case + "__edges"])


@pytest.mark.parametrize("seed", range(4))
def test_mixed_streams_vs_oracle(torch_cuda, seed):
    recs = S.mixed_stream(300, seed + 100)
    # the oracle and the GPU agree on every stream (the reference itself diverges where matrix
    # tiles wrap the leading dimension; tests/golden/wrap_golden.npz pins that difference)
    np.testing.assert_array_equal(gpu_edges(recs), U.oracle_edges(recs))


_WRAP = np.load(os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden", "wrap_golden.npz"))


@pytest.mark.parametrize("case", sorted(k[:-len("__stream")] for k in _WRAP.files if k.endswith("__stream")))
def test_wrapped_tiles_gpu_edges_are_the_pinned_pointwise_set(torch_cuda, case):
    """On streams with tiles that wrap the leading dimension the GPU resolver gives exactly the
    point-wise edge set the fixture records beside the reference's (their difference is pinned
    by tests/test_oracle.py)."""
    np.testing.assert_array_equal(gpu_edges(_WRAP[case + "__stream"]), _WRAP[case + "__pointwise_edges"])


def test_microbench_16k_vs_oracle(torch_cuda):
    recs = S.microbench_stream(16384, 12345)
    np.testing.assert_array_equal(gpu_edges(recs, batches=3), U.oracle_edges(recs))


def test_heat_graph_100_steps_vs_oracle(torch_cuda):
    recs = S.heat_stream(1024, 1024, 128, 128, 100)
    np.testing.assert_array_equal(gpu_edges(recs, batches=5), U.oracle_edges(recs))


@pytest.mark.parametrize("which", ["microbench_32k", "heat_4096_t64_s10"])
def test_large_matrix_batches_vs_oracle(torch_cuda, which):
    # a small first batch creates the domain; the large second batch (tens of thousands of
    # matrix records on existing domains) is split over host threads when building ops
    recs = S.microbench_stream(32768, 777) if which == "microbench_32k" else S.heat_stream(4096, 4096, 64, 64, 10)
    cut = int(np.searchsorted(recs["task"], 500))
    r = xk.Resolver()
    r.add(recs[:cut]); r.add(recs[cut:])
    e = r.edges()
    r.close()
    np.testing.assert_array_equal(e, U.oracle_edges(recs))


def test_many_readers(torch_cuda):
    # 150 readers of the same rows, then a writer: the writer depends on all 150 readers
    tasks = [[("m", S.W, 1 << 20, 256, 0, 0, 64, 8, 8)]]
    tasks += [[("m", S.R, 1 << 20, 256, 0, 0, 64, 8, 8)] for _ in range(150)]
    tasks += [[("m", S.W, 1 << 20, 256, 16, 2, 8, 2, 8)]]
    recs = S.from_tuples(tasks)
    e = gpu_edges(recs)
    np.testing.assert_array_equal(e, U.oracle_edges(recs))
    assert sum(1 for p, s in e if s == 151) == 150


@pytest.mark.parametrize("nreaders,batches", [(5000, 1), (3000, 9)])
def test_thousands_of_readers_spill(torch_cuda, nreaders, batches):
    # far more readers of one region than a cell keeps inline (they spill to chained chunks,
    # across batches too); then two writers, each over part of it, depend on every reader
    tasks = [[("m", S.W, 1 << 20, 256, 0, 0, 64, 8, 8)]]
    tasks += [[("m", S.R, 1 << 20, 256, 0, 0, 64, 8, 8)] for _ in range(nreaders)]
    tasks += [[("m", S.W, 1 << 20, 256, 16, 2, 8, 2, 8)], [("m", S.W, 1 << 20, 256, 40, 5, 4, 1, 8)]]
    recs = S.from_tuples(tasks)
    e = gpu_edges(recs, batches, seed=3)
    np.testing.assert_array_equal(e, U.oracle_edges(recs))
    assert sum(1 for p, s in e if s == nreaders + 1) == nreaders


def test_spilled_readers_survive_refinement(torch_cuda):
    # readers spill in a first batch; the second batch brings new boundaries that split the
    # cells (each piece copies the spilled readers), appends readers to some pieces, and then
    # writes each piece separately
    ld, base = 512, 1 << 22
    first = [[("m", S.W, base, ld, 0, 0, 256, 16, 8)]]
    first += [[("m", S.R, base, ld, 0, 0, 256, 16, 8)] for _ in range(200)]
    second = [[("m", S.R, base, ld, 64, 4, 32, 4, 8)] for _ in range(40)]
    second += [[("m", S.W, base, ld, x, y, 16, 3, 8)] for x in (0, 60, 100, 200) for y in (0, 5, 12)]
    recs = S.from_tuples(first + second)
    cut = int(np.searchsorted(recs["task"], len(first)))
    r = xk.Resolver()
    r.add(recs[:cut]); r.add(recs[cut:])
    e = r.edges()
    r.close()
    np.testing.assert_array_equal(e, U.oracle_edges(recs))


class _DevView:
    """Wraps a raw device pointer for torch.as_tensor (CUDA array interface)."""
    def __init__(self, ptr, n):
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": "<i4", "data": (ptr, False), "version": 3}


def test_graph_csr_consistent(torch_cuda):
    torch = torch_cuda
    recs = S.microbench_stream(3000, 5, n=2048, ld=2048)
    r = xk.Resolver()
    r.add(recs)
    g = r.graph()
    nt, ne = g.ntasks, g.nedges
    ptr = torch.as_tensor(_DevView(g.succ_ptr, nt + 1), device="cuda").cpu().numpy()
    succ = torch.as_tensor(_DevView(g.succ, ne), device="cuda").cpu().numpy()
    npred = torch.as_tensor(_DevView(g.npred, nt), device="cuda").cpu().numpy()
    e = U.oracle_edges(recs)
    assert ne == len(e) and ptr[-1] == ne and ptr[0] == 0
    np.testing.assert_array_equal(np.diff(ptr), np.bincount(e[:, 0], minlength=nt))
    np.testing.assert_array_equal(npred, np.bincount(e[:, 1], minlength=nt))
    pairs = np.stack([np.repeat(np.arange(nt), np.diff(ptr)), succ], axis=1)
    np.testing.assert_array_equal(pairs, e)
    r.close()


def test_rejects_bad_streams(torch_cuda):
    r = xk.Resolver()
    bad = S.from_tuples([[("m", S.R, 4096, 64, 0, 0, 8, 8, 8)], [("m", S.W, 4096, 64, 0, 0, 8, 8, 8)]])
    bad["task"][1] = 5                       # task ids must be dense
    with pytest.raises(xk.XkbError):
        r.add(bad)
    bad2 = S.from_tuples([[("m", 0, 4096, 64, 0, 0, 8, 8, 8)]])    # mode 0
    with pytest.raises(xk.XkbError):
        r.add(bad2)
    bad3 = S.from_tuples([[("h", S.W, 4096)]])
    bad3["reserved"] = 4 << 8                # a concurrent access that was not expanded
    with pytest.raises(xk.XkbError) as ei:
        r.add(bad3)
    assert "xkb_handle_map_expand" in str(ei.value)
    ok = S.from_tuples([[("m", S.W, 4096, 64, 0, 0, 8, 8, 8)], [("m", S.R, 4096, 64, 0, 0, 8, 8, 8)]])
    r.add(ok)
    np.testing.assert_array_equal(r.edges(), [[0, 1]])
    r.close()


def _readers_stream(nreaders):
    tasks = [[("m", S.W, 1 << 20, 256, 0, 0, 64, 8, 8)]]
    tasks += [[("m", S.R, 1 << 20, 256, 0, 0, 64, 8, 8)] for _ in range(nreaders)]
    tasks += [[("m", S.W, 1 << 20, 256, 16, 2, 8, 2, 8)], [("m", S.W, 1 << 20, 256, 40, 5, 4, 1, 8)]]
    tasks += [[("m", S.R, 1 << 20, 256, 0, 0, 64, 8, 8)] for _ in range(nreaders // 2)]
    tasks += [[("m", S.RW, 1 << 20, 256, 0, 0, 64, 8, 8)]]
    return S.from_tuples(tasks)


@pytest.mark.parametrize("nseg,global_bins", [(2, False), (3, True), (8, False), (1, True)])
def test_time_split_resolution_same_edges(torch_cuda, monkeypatch, nseg, global_bins):
    """Every region's op list cut into nseg segments (XKB_RESOLVE_SEGMENTS forces the time-split
    kernels: one pass of PUT ops writing the state at each cut, then one CTA per region and
    segment emitting its LINK ops' edges): the reference's golden edges, the oracle's edges on
    seeded streams and in several batches, and reader lists past the inline ones (spilled before a
    cut, across cuts, added inside a segment, over several batches) give the same edge sets; with
    the global-atomic binning too (what domains of more than 12,288 regions use)."""
    monkeypatch.setenv("XKB_RESOLVE_SEGMENTS", str(nseg))
    if global_bins:                     # the binning without block-local counts (domains of many regions)
        monkeypatch.setenv("XKB_RESOLVE_BIN_GLOBAL", "1")
    for case in CASES:
        np.testing.assert_array_equal(gpu_edges(expanded(GOLDEN[case + "__stream"])), GOLDEN[case + "__edges"], err_msg=case)
    for case in ("heat_1024_t128_s3", "microbench_1024_2000", "mixed_segmat_0"):
        np.testing.assert_array_equal(gpu_edges(GOLDEN[case + "__stream"], 3, seed=nseg), GOLDEN[case + "__edges"], err_msg=case)
    for seed in range(2):
        recs = S.mixed_stream(300, seed + 100)
        np.testing.assert_array_equal(gpu_edges(recs), U.oracle_edges(recs))
    recs = S.microbench_stream(16384, 12345)
    np.testing.assert_array_equal(gpu_edges(recs), U.oracle_edges(recs))
    for nreaders, batches in ((100, 1), (3000, 1), (3000, 4)):
        recs = _readers_stream(nreaders)
        np.testing.assert_array_equal(gpu_edges(recs, batches, seed=7), U.oracle_edges(recs), err_msg=f"{nreaders} readers")


@pytest.mark.parametrize("nseg", [1, 5, 24])
@pytest.mark.parametrize("writers", [0, 3, 60])
def test_segments_look_back(torch_cuda, monkeypatch, nseg, writers):
    """Segments find each cell's last write by looking back from their cut: streams whose cells are
    never written, written a few times far back, and often, over two batches, give the oracle's edges."""
    monkeypatch.setenv("XKB_RESOLVE_SEGMENTS", str(nseg))
    rng = np.random.default_rng(10 * nseg + writers)
    tasks = []
    for t in range(1200):
        x, y, m, n = (int(v) for v in (rng.integers(0, 12) * 16, rng.integers(0, 12) * 16, rng.integers(1, 5) * 16, rng.integers(1, 5) * 16))
        w = writers and t % (1200 // writers) == 0
        tasks.append([("m", S.RW if w and t % 2 else S.W if w else S.R, 1 << 20, 256, x, y, m, n, 8)])
    recs = S.from_tuples(tasks)
    want = U.oracle_edges(recs)
    for batches in (1, 2):
        np.testing.assert_array_equal(gpu_edges(recs, batches, seed=5), want)


@pytest.mark.parametrize("nreaders", [1, 31, 32, 33, 511, 512, 513, 1500])
def test_successor_lists_ascending(torch_cuda, nreaders):
    """A writer followed by nreaders readers of its cells: its successor list comes back in ascending
    order whatever sorts it (one warp's registers, shared memory, global memory)."""
    torch = torch_cuda
    recs = S.from_tuples([[("m", S.W, 1 << 20, 256, 0, 0, 64, 8, 8)]] +
                         [[("m", S.R, 1 << 20, 256, 8 * (k % 8), 0, 8, 8, 8)] for k in range(nreaders)])
    r = xk.Resolver()
    r.add(recs)
    g = r.graph()
    assert g.nedges == nreaders
    succ = torch.as_tensor(_DevView(g.succ, g.nedges), device="cuda").cpu().numpy()
    np.testing.assert_array_equal(succ, np.arange(1, nreaders + 1))
    r.close()


def diagonal(cells, first_task, count, passes=1):
    """Write accesses to the first `count` of the `cells` 64 x 64 blocks on the diagonal of a matrix, a
    task each, `passes` times over: 64 (cells / 8)^2 regions in the domain once all blocks were named."""
    k = np.tile(np.arange(count, dtype=np.uint64), passes)
    r = np.zeros(len(k), dtype=S.REC)
    r["task"] = first_task + np.arange(len(k))
    r["type"], r["mode"], r["ld"], r["sizeof_type"], r["m"], r["n"] = S.MATRIX, S.RW, 64 * cells, 8, 64, 64
    r["offset_m"] = r["offset_n"] = 64 * k
    return r


def run_logged(tmp_path, body, **env):
    """Run `body` (Python, with diagonal() and mark(text) at hand) in a process whose calls of the CUDA
    runtime are logged (tests/cpp/cudart_log.c); the log's lines, split."""
    tests = os.path.dirname(os.path.abspath(__file__))
    shim, log = str(tmp_path / "cudart_log.so"), str(tmp_path / "log.txt")
    subprocess.run(["gcc", "-O1", "-Wall", "-Werror", "-shared", "-fPIC", os.path.join(tests, "cpp", "cudart_log.c"), "-o", shim, "-ldl"],
                   check=True)
    code = (f"import sys, ctypes; sys.path[:0] = [{tests!r}, {U.REPO!r}]\n"
            "import numpy as np, xkaapi_b200 as xk\nfrom test_resolver_gpu import diagonal\n"
            f"mark = lambda text: ctypes.CDLL({shim!r}).cudart_log_mark(text.encode())\n" + body)
    r = subprocess.run([sys.executable, "-c", code], env=dict(os.environ, LD_PRELOAD=shim, CUDART_LOG=log, **env),
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    return [ln.split() for ln in open(log).read().splitlines()]


def test_shared_memory_limits_are_never_lowered(torch_cuda, tmp_path):
    """A kernel's shared-memory limit belongs to the process: a batch that needs less must not lower it
    below what another thread's batch is about to launch with."""
    log = run_logged(tmp_path, """
big, small = xk.Resolver(), xk.Resolver()
big.add(diagonal(870, 0, 870, 800))        # 11,881 regions, 1.4 M ops: more than one bitmap of 160 KB
small.add(diagonal(640, 0, 640, 320))      # 6,400 regions, 410,000 ops
""")
    limits = {}
    for ln in log:
        if ln[0] == "smem":
            assert int(ln[2]) >= limits.get(ln[1], 0), log
            limits[ln[1]] = int(ln[2])
    assert len(limits) >= 2


def test_region_lists_sorted_over_several_bitmaps(torch_cuda):
    """1.4 M ops, more than one bitmap of the list sort holds, in lists of 12,800: every block's writes
    follow one another."""
    n = 870 * 800
    t = np.arange(n - 870)
    np.testing.assert_array_equal(gpu_edges(diagonal(870, 0, 870, 800)), np.stack([t, t + 870], axis=1))


@pytest.mark.parametrize("cache,blocks,passes", [("0", 40, 3), ("1", 870, 7900)])
def test_blocks_that_are_not_kept_stay_with_their_resolver(torch_cuda, tmp_path, cache, blocks, passes):
    """Page-locked blocks that would be unlocked when a batch gives them back -- all of them where none
    is kept, those over 256 MB (6.9 M rects) otherwise -- serve the resolver's next batch, and
    go with the resolver."""
    log = run_logged(tmp_path, f"""
r = xk.Resolver()
for k in range(2):
    r.add(diagonal({blocks}, k * {blocks * passes}, {blocks}, {passes}))
    mark("added")
assert r.graph().nedges == {blocks * (2 * passes - 1)}
r.close()
mark("closed")
""", XKB_POOL_CACHE=cache)
    added = [k for k, ln in enumerate(log) if ln == ["added"]]
    assert any(ln[0] == "lock" for ln in log[:added[0]])
    assert not [ln for ln in log[added[0]:added[1]] if ln[0] in ("lock", "unlock")], log
    freed = {ln[1] for ln in log[added[1]:log.index(["closed"])] if ln[0] == "unlock"}
    largest = max((int(ln[2]), ln[1]) for ln in log if ln[0] == "lock")
    assert largest[1] in freed, log


def test_memory_kept_for_the_next_resolver_ends_with_its_context(torch_cuda, tmp_path):
    """The page-locked blocks and the device pool kept for the next resolver are not handed out after
    cudaDeviceReset has ended their context: the next resolver locks blocks of its own, and works."""
    log = run_logged(tmp_path, """
cudart = ctypes.CDLL("libcudart.so.12")
for k in range(3):
    r = xk.Resolver()
    r.add(diagonal(40, 0, 40, 500))
    assert r.graph().nedges == 40 * 499
    e = r.edges()
    np.testing.assert_array_equal(e, np.stack([np.arange(len(e)), np.arange(len(e)) + 40], axis=1))
    r.close()
    mark("closed")
    if k == 1:
        assert cudart.cudaDeviceReset() == 0
""")
    closed = [k for k, ln in enumerate(log) if ln == ["closed"]]
    locks = [sorted(int(ln[2]) for ln in part if ln[0] == "lock")
             for part in (log[:closed[0]], log[closed[0]:closed[1]], log[closed[1]:])]
    assert locks[0] and locks[1] == [] and locks[2] == locks[0], log
    assert not [ln for ln in log[closed[1]:] if ln[0] == "unlock"], log


def test_page_locked_memory_is_given_back_with_the_last_resolver(torch_cuda, tmp_path):
    """Blocks kept for the next batch are unlocked when the last resolver goes, all but 64 MB."""
    log = run_logged(tmp_path, """
first, second = xk.Resolver(), xk.Resolver()
first.add(diagonal(870, 0, 870, 2000))             # 70 MB of rects: a block of 128 MB
first.close()
mark("one")
second.add(diagonal(40, 0, 40, 3))
second.close()
mark("none")
""")
    sizes = {ln[1]: int(ln[2]) for ln in log if ln[0] == "lock"}
    left = log.index(["one"])
    assert max(sizes.values()) == 128 << 20
    assert not [ln for ln in log[:left] if ln[0] == "unlock"], log
    held = sum(sizes.values()) - sum(sizes[ln[1]] for ln in log if ln[0] == "unlock" and ln[1] in sizes)
    assert held <= 64 << 20, log

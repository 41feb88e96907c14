"""GPU parity of the brute-force matcher (CUDA path via the C ABI) against the CPU oracle.

Bar: bit-exact indices and distances in both directions (reference tie-break: lowest index),
bit-exact second-best distance and flags (oracle-pinned extension).
"""
import numpy as np
import pytest
import torch

from rapidsfm_b200 import synth

pytestmark = pytest.mark.gpu


def _dev(x):
    return torch.from_numpy(np.ascontiguousarray(x)).cuda()


def _run_ext(rsfm, pairs):
    tasks = [rsfm.BFTask(_dev(a), _dev(b)) for a, b in pairs]
    rsfm.bf_match_ext(tasks)
    torch.cuda.synchronize()
    assert rsfm.device_error() == 0
    out = []
    for t in tasks:
        fi, fd = rsfm.unpack_best(t.bestA)
        bi, bd = rsfm.unpack_best(t.bestB)
        out.append((np.stack([fi, fd], 1), np.stack([bi, bd], 1),
                    t.secondA.cpu().numpy().view(np.uint32), t.flagsA.cpu().numpy().view(np.uint32)))
    return out


def _check(oracle, a, b, got):
    fwd, bwd, sec, flags = got
    efwd, ebwd, esec = oracle.bf_match(a, b)
    eflags = oracle.match_flags(efwd, esec, ebwd)
    np.testing.assert_array_equal(fwd, efwd)
    np.testing.assert_array_equal(bwd, ebwd)
    np.testing.assert_array_equal(sec, esec)
    np.testing.assert_array_equal(flags, eflags)


def test_sqr_norm(rsfm, oracle):
    d = synth.uniform_bytes(1000, 5)
    got = rsfm.precomp_sift_sqr_norm(_dev(d)).cpu().numpy().view(np.uint32)
    np.testing.assert_array_equal(got, oracle.sqr_norm(d))


def test_uniform_897(rsfm, oracle):
    # Shape of the reference's own kernel test (test/bruteForceMatchKernelTest.cpp:300: 897 x 897).
    a = synth.uniform_bytes(897, 1)
    b = synth.uniform_bytes(897, 2)
    _check(oracle, a, b, _run_ext(rsfm, [(a, b)])[0])


def test_sift_config0(rsfm, oracle):
    q, t, _ = synth.make_pair(4096, 4096, 0.6, 8.0, seed=0)
    _check(oracle, q, t, _run_ext(rsfm, [(q, t)])[0])


@pytest.mark.parametrize("na,nb", [(1, 1), (1, 300), (300, 1), (129, 127), (2000, 5000), (1100, 130), (5, 4097)])
def test_ragged(rsfm, oracle, na, nb):
    q, t, _ = synth.make_pair(na, nb, 0.5, 6.0, seed=na * 7 + nb)
    _check(oracle, q, t, _run_ext(rsfm, [(q, t)])[0])


def test_ties_lowest_index(rsfm, oracle):
    # Heavy ties: 40 distinct descriptors repeated; every row/column has many equal minima.
    base = synth.uniform_bytes(40, 3)
    rng = np.random.default_rng(0)
    a = base[rng.integers(0, 40, 700)]
    b = base[rng.integers(0, 40, 900)]
    _check(oracle, a, b, _run_ext(rsfm, [(a, b)])[0])


def test_extreme_values(rsfm, oracle):
    # All-0 and all-255 descriptors reach the largest distance 128*255^2.
    a = np.zeros((260, 128), np.uint8)
    a[::2] = 255
    b = np.zeros((300, 128), np.uint8)
    b[1::3] = 255
    b[2::3, :64] = 255
    _check(oracle, a, b, _run_ext(rsfm, [(a, b)])[0])


def test_many_tasks(rsfm, oracle):
    # More than the 16 tasks per launch: the host chunks them like the reference launcher.
    pairs = []
    for k in range(19):
        q, t, _ = synth.make_pair(100 + 37 * k, 90 + 53 * k, 0.4, 5.0, seed=100 + k)
        pairs.append((q, t))
    got = _run_ext(rsfm, pairs)
    for (a, b), g in zip(pairs, got):
        _check(oracle, a, b, g)


def test_empty_sides(rsfm, oracle):
    a = synth.uniform_bytes(50, 1)
    e = np.zeros((0, 128), np.uint8)
    fwd, bwd, sec, flags = _run_ext(rsfm, [(a, e)])[0]
    assert (fwd == 0xFFFFFFFF).all() and len(bwd) == 0
    assert (flags == 0).all()


def test_reference_api_matches_ext(rsfm, oracle):
    q, t, _ = synth.make_pair(3000, 2500, 0.5, 8.0, seed=11)
    task = rsfm.BFTask(_dev(q), _dev(t))
    rsfm.bf_match([task])
    torch.cuda.synchronize()
    fi, fd = rsfm.unpack_best(task.bestA)
    bi, bd = rsfm.unpack_best(task.bestB)
    efwd, ebwd, _ = oracle.bf_match(q, t)
    np.testing.assert_array_equal(np.stack([fi, fd], 1), efwd)
    np.testing.assert_array_equal(np.stack([bi, bd], 1), ebwd)


def test_full_size_exact(rsfm, oracle):
    # The dense-contraction workload itself (32768 x 32768, 50 % overlap, noise 10, seed 1: the
    # pair bench.py times): every forward match, second-best distance, flag word and backward
    # match against the oracle's exhaustive loop (test/bruteForceMatchKernelTest.cpp:140-164 with
    # the (distance, index) tie rule of bruteForceMatch.cuh:110-187).
    q, t, _ = synth.make_pair(32768, 32768, 0.5, 10.0, seed=1)
    _check(oracle, q, t, _run_ext(rsfm, [(q, t)])[0])


def test_full_size_reference_entry(rsfm, oracle):
    # Same pair through the reference-shaped entry point (rsfm_bf_match, no extension outputs).
    q, t, _ = synth.make_pair(32768, 32768, 0.5, 10.0, seed=1)
    task = rsfm.BFTask(_dev(q), _dev(t))
    rsfm.bf_match([task])
    torch.cuda.synchronize()
    assert rsfm.device_error() == 0
    fi, fd = rsfm.unpack_best(task.bestA)
    bi, bd = rsfm.unpack_best(task.bestB)
    efwd, ebwd, _ = oracle.bf_match(q, t)
    np.testing.assert_array_equal(np.stack([fi, fd], 1), efwd)
    np.testing.assert_array_equal(np.stack([bi, bd], 1), ebwd)


def test_uniform_large_exact(rsfm, oracle):
    # Uniform random bytes (norms spread over a wide range, unlike SIFT-like rows) at a size with
    # many units per row and column: 12288 x 9000.
    a = synth.uniform_bytes(12288, 21)
    b = synth.uniform_bytes(9000, 22)
    _check(oracle, a, b, _run_ext(rsfm, [(a, b)])[0])


def _norm_spread(n, seed):
    """SIFT-like rows among all-zero, all-127 and (odd seeds) all-255 and all-128 ones: norms beyond
    what the norm digits hold, and units that may and may not be doubled (a byte above 127)."""
    d = np.minimum(synth.make_pair(n, 1, 0.0, 1.0, seed=seed)[0], 127)
    d[::97] = 0
    d[5::89] = 127
    if seed % 2:
        d[3::83] = 255
        d[7::101] = 128
    return d


@pytest.mark.parametrize("na,nb", [(1, 17), (15, 16), (127, 128), (128, 129), (255, 257), (256, 256), (257, 511),
                                   (513, 4097), (64, 9000), (2500, 300)])
@pytest.mark.parametrize("seed", [2, 3])
def test_unit_and_chunk_edges(rsfm, oracle, na, nb, seed):
    # Around the 16-value chunks, 128-row halves, 256-row units and 256-column blocks; norms outside
    # the digits' range (residuals) and both kinds of units (doubled rows, rows with large bytes).
    a, b = _norm_spread(na, seed), _norm_spread(nb, seed + 2)
    _check(oracle, a, b, _run_ext(rsfm, [(a, b)])[0])


@pytest.mark.parametrize("sizes", [[(700, 900), (300, 0), (0, 40), (1000, 20)], [(9000, 9100), (30, 8000)]])
def test_phases_in_one_launch_and_apart(rsfm, oracle, sizes):
    # A call is init, match and resolution, with the flags in it. Same results from both entry
    # points, empty sides.
    pairs = []
    for k, (na, nb) in enumerate(sizes):
        q, t, _ = synth.make_pair(max(na, 1), max(nb, 1), 0.5, 8.0, seed=500 + k)
        pairs.append((q[:na], t[:nb]))
    tasks = [rsfm.BFTask(_dev(a), _dev(b)) for a, b in pairs]
    rsfm.bf_match_ext(tasks)
    assert rsfm.last_launch_count() == 3
    got = _run_ext(rsfm, pairs)
    rsfm.bf_match(tasks)
    for (a, b), g, t in zip(pairs, got, tasks):
        if len(a) and len(b):
            _check(oracle, a, b, g)
        else:
            assert (g[0] == 0xFFFFFFFF).all() and (g[1] == 0xFFFFFFFF).all() and (g[3] == 0).all()
        np.testing.assert_array_equal(np.stack(rsfm.unpack_best(t.bestA), 1), g[0])
        np.testing.assert_array_equal(np.stack(rsfm.unpack_best(t.bestB), 1), g[1])


def test_user_graph_capture_and_streams(rsfm, oracle):
    # A caller's own graph around a small call (launches that overlap), and calls on two streams at once.
    pairs = [synth.make_pair(800, 1000, 0.5, 8.0, seed=40)[:2], synth.make_pair(1200, 600, 0.5, 8.0, seed=41)[:2]]
    tasks = [rsfm.BFTask(_dev(a), _dev(b)) for a, b in pairs]
    rsfm.bf_match_ext(tasks)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        rsfm.bf_match_ext([tasks[0]])
    for t in tasks:  # all that the replays and the direct calls have to write
        for out in (t.bestA, t.bestB, t.secondA, t.flagsA):
            out.fill_(0x55)
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in range(2)]
    for _ in range(5):
        with torch.cuda.stream(streams[0]):
            graph.replay()
        rsfm.bf_match_ext([tasks[1]], stream=streams[1])
    torch.cuda.synchronize()
    assert rsfm.device_error() == 0
    for (a, b), t in zip(pairs, tasks):
        got = (np.stack(rsfm.unpack_best(t.bestA), 1), np.stack(rsfm.unpack_best(t.bestB), 1),
               t.secondA.cpu().numpy().view(np.uint32), t.flagsA.cpu().numpy().view(np.uint32))
        _check(oracle, a, b, got)


@pytest.mark.parametrize("na,nb", [(64, 20000), (20000, 64), (1, 5000), (5000, 1), (75400, 300), (75600, 300), (300, 75600)])
def test_few_blocks_many_results(rsfm, oracle, na, nb):
    # Long thin pairs: little matching, many results, and no launch more than a square pair's. The flags
    # are a launch of their own only beyond 128 groups of four results per SM.
    a, b = synth.make_pair(na, nb, 0.5, 8.0, seed=na + 2 * nb)[:2]
    task = rsfm.BFTask(_dev(a), _dev(b))
    rsfm.bf_match_ext([task])
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert rsfm.last_launch_count() == (3 if (na + nb + 3) // 4 <= 128 * sms else 4)
    _check(oracle, a, b, _run_ext(rsfm, [(a, b)])[0])


@pytest.mark.parametrize("na,nb,seed", [(200, 150, 0), (3000, 2500, 1), (20000, 9000, 2)])
def test_cross_check_among_equal_rows_of_a_chunk(rsfm, oracle, na, nb, seed):
    """Runs of equal rows (1 to 24 long, so inside a 16-row chunk and across its edges): of the rows that
    are as close to a column only the first is its match. Columns whose index is resolved before or after
    the row that looks it up give the same flags, call after call."""
    rng = np.random.default_rng(seed)
    base = synth.make_pair(na, 1, 0.0, 1.0, seed=seed)[0]
    a = np.repeat(base, rng.integers(1, 25, na), axis=0)[:na]
    b = np.minimum(a[rng.integers(0, na, nb)] + (rng.random((nb, 128)) < 0.05 * rng.integers(0, 2, (nb, 1))), 255)
    b = b.astype(np.uint8)
    efwd, ebwd, esec = oracle.bf_match(a, b)
    eflags = oracle.match_flags(efwd, esec, ebwd)
    assert 0 < (eflags & 2).sum() < 2 * na
    for _ in range(3):
        fwd, bwd, sec, flags = _run_ext(rsfm, [(a, b)])[0]
        np.testing.assert_array_equal(fwd, efwd)
        np.testing.assert_array_equal(bwd, ebwd)
        np.testing.assert_array_equal(sec, esec)
        np.testing.assert_array_equal(flags, eflags)


def test_stream_of_a_green_context(rsfm, oracle):
    """A stream that owns 16 SMs: a call may not need all its blocks resident at once."""
    cu = pytest.importorskip("cuda.bindings.driver")

    def ok(r):
        assert r[0] == cu.CUresult.CUDA_SUCCESS, r[0]
        return r[1] if len(r) == 2 else r[1:]

    torch.cuda.synchronize()  # (the primary context is there and current)
    dev = ok(cu.cuDeviceGet(torch.cuda.current_device()))
    sms = ok(cu.cuDeviceGetDevResource(dev, cu.CUdevResourceType.CU_DEV_RESOURCE_TYPE_SM))
    groups, _, _ = ok(cu.cuDevSmResourceSplitByCount(1, sms, 0, 16))
    desc = ok(cu.cuDevResourceGenerateDesc(groups[:1], 1))
    green = ok(cu.cuGreenCtxCreate(desc, dev, cu.CUgreenCtxCreate_flags.CU_GREEN_CTX_DEFAULT_STREAM))
    raw = ok(cu.cuGreenCtxStreamCreate(green, cu.CUstream_flags.CU_STREAM_NON_BLOCKING, 0))
    try:
        stream = torch.cuda.ExternalStream(int(raw))
        a, b = synth.make_pair(3000, 2500, 0.5, 8.0, seed=77)[:2]
        task = rsfm.BFTask(_dev(a), _dev(b))
        torch.cuda.synchronize()
        rsfm.bf_match_ext([task], stream=stream)
        stream.synchronize()
        got = (np.stack(rsfm.unpack_best(task.bestA), 1), np.stack(rsfm.unpack_best(task.bestB), 1),
               task.secondA.cpu().numpy().view(np.uint32), task.flagsA.cpu().numpy().view(np.uint32))
        _check(oracle, a, b, got)
    finally:
        ok(cu.cuStreamDestroy(raw))
        ok(cu.cuGreenCtxDestroy(green))


def test_calls_whose_kernels_overlap(rsfm, oracle):
    """A call's kernels start while the one before them runs. Calls one after the other without a wait,
    on inputs written by a kernel just before each and into the same buffers, in all three forms (norms
    and 4-bit widening right before the match): every result as if the call were alone."""
    n = [(300, 900), (900, 300), (2300, 1200), (40, 5000)]
    pairs = [[synth.make_pair(na, nb, 0.5, 8.0, seed=800 + 10 * k + r)[:2] for r in range(3)] for k, (na, nb) in enumerate(n)]
    src = [[(_dev(a), _dev(b)) for a, b in p] for p in pairs]
    bufs = [(torch.empty_like(p[0][0]), torch.empty_like(p[0][1])) for p in src]
    got = []
    for rep in range(4):
        for k, (a, b) in enumerate(bufs):
            for r in range(3):
                a.copy_(src[k][r][0])
                b.copy_(src[k][r][1])
                ext, idp = rsfm.BFTask(a, b), rsfm.BFTask(a, b, norms=False)
                rsfm.bf_match_ext([ext])
                rsfm.bf_match_idp([idp])
                four = rsfm.BFTask(rsfm.sift_desc_8b_to_4b(a), rsfm.sift_desc_8b_to_4b(b), bits=4)
                rsfm.bf_match_4b([four])
                got.append((k, r, ext, idp, four))
    torch.cuda.synchronize()
    assert rsfm.device_error() == 0
    want = {}
    for k, r, ext, idp, four in got:
        a, b = pairs[k][r]
        if (k, r) not in want:
            fwd, bwd, sec = oracle.bf_match(a, b)
            want[k, r] = (fwd, bwd, sec, oracle.match_flags(fwd, sec, bwd), oracle.bf_match(
                oracle.desc_4b_values(oracle.desc_8b_to_4b(a)), oracle.desc_4b_values(oracle.desc_8b_to_4b(b))))
        fwd, bwd, sec, flags, w4 = want[k, r]
        for t, (f, g) in ((ext, (fwd, bwd)), (idp, (fwd, bwd)), (four, w4[:2])):
            np.testing.assert_array_equal(np.stack(rsfm.unpack_best(t.bestA), 1), f)
            np.testing.assert_array_equal(np.stack(rsfm.unpack_best(t.bestB), 1), g)
        np.testing.assert_array_equal(ext.secondA.cpu().numpy().view(np.uint32), sec)
        np.testing.assert_array_equal(ext.flagsA.cpu().numpy().view(np.uint32), flags)


def test_default_stream_is_the_current_one(rsfm):
    # Without a stream argument a call goes to torch's current stream of the current device.
    from rapidsfm_b200.matcher import _stream_ptr
    assert _stream_ptr(None).value == (torch.cuda.current_stream().cuda_stream or None)
    for priority in (0, -1):
        s = torch.cuda.Stream(priority=priority)
        with torch.cuda.stream(s):
            assert _stream_ptr(None).value == s.cuda_stream == _stream_ptr(s).value
    assert _stream_ptr(None).value == (torch.cuda.current_stream().cuda_stream or None)


def test_second_context_of_the_device(rsfm, oracle):
    """What the library keeps between calls belongs to a context: after calls in the primary one, a
    call in another context of the same device uses that context's variables and kernel attributes."""
    cu = pytest.importorskip("cuda.bindings.driver")

    def ok(r):
        assert r[0] == cu.CUresult.CUDA_SUCCESS, r[0]
        return r[1] if len(r) == 2 else None

    a, b = synth.make_pair(700, 900, 0.5, 8.0, seed=91)[:2]
    _check(oracle, a, b, _run_ext(rsfm, [(a, b)])[0])  # (primary context)
    lib = rsfm._lib.load()
    efwd, ebwd, _ = oracle.bf_match(a, b)
    ctx = ok(cu.cuCtxCreate(0, ok(cu.cuDeviceGet(torch.cuda.current_device()))))
    try:
        bufs = []
        for x in (a, b, oracle.sqr_norm(a), oracle.sqr_norm(b), np.zeros((len(a), 2), np.uint32), np.zeros((len(b), 2), np.uint32)):
            x = np.ascontiguousarray(x)
            p = ok(cu.cuMemAlloc(x.nbytes))
            ok(cu.cuMemcpyHtoD(p, x.ctypes.data, x.nbytes))
            bufs.append((int(p), x))
        (pa, _), (pb, _), (na, _), (nb, _), (ra, fwd), (rb, bwd) = bufs
        task = (rsfm._lib.SiftBFTask * 1)(rsfm._lib.SiftBFTask(len(a), len(b), pa, pb, ra, rb, na, nb))
        rsfm._lib.check(lib.rsfm_bf_match(task, 1, None), "rsfm_bf_match")
        assert rsfm.device_error() == 0
        ok(cu.cuCtxSynchronize())
        ok(cu.cuMemcpyDtoH(fwd.ctypes.data, ra, fwd.nbytes))
        ok(cu.cuMemcpyDtoH(bwd.ctypes.data, rb, bwd.nbytes))
    finally:
        ok(cu.cuCtxDestroy(ctx))
    np.testing.assert_array_equal(fwd, efwd)
    np.testing.assert_array_equal(bwd, ebwd)
    _check(oracle, a, b, _run_ext(rsfm, [(a, b)])[0])  # (the primary one again)

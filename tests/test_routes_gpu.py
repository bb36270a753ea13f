"""The routes a gemv / gemm / sum-of-squares call takes by its sizes, alignment and type, each at
the sizes where it can go wrong, bit for bit against the oracle: gemm tiles cut between CTAs (and
the whole-tile fallback when their scratch cannot be had), K blocks that leave the unchecked
path (non-finite products, the top bin, zero rows, raises in a late block), gemv rows that
start at every 4-byte alignment, matrices with fewer rows than alignment phases, both sides
of the direct kernels' size limits, scales that grow inside and between warps, and the int8
digits of magnitudes far below their row's largest."""
import numpy as np
import pytest

from _cmp import same_bits, same_state, same_value
from _data import gen, gen_complex
from _ffi import binned_zeros, ptr
from _xblas import lib_gemm, lib_gemv, rb_gemm, rb_gemv

pytestmark = pytest.mark.gpu

REAL = {"d": np.float64, "s": np.float32, "z": np.float64, "c": np.float32}
FULL = {"d": np.float64, "s": np.float32, "z": np.complex128, "c": np.complex64}


def ops(t, n, seed, dist="uniform"):
    return gen(dist, n, seed, REAL[t]) if t in "ds" else gen_complex(dist, n, seed, FULL[t])


def dev(cuda, a):
    return cuda.from_numpy(np.ascontiguousarray(a).view(a.real.dtype)).cuda()


def scalars(t):
    return (1.5, 0.5) if t in "ds" else (1.5 - 0.25j, 0.5 + 0.125j)


def oracle_gemm(port, t, fold, ta, tb, M, N, K, A, lda, B, ldb, C, ldc):
    al, be = scalars(t)
    if t == "d":
        port.rdgemm(fold, b"r", ta.encode(), tb.encode(), M, N, K, al, ptr(A), lda, ptr(B), ldb, be,
                    ptr(C), ldc)
    else:
        lib_gemm(port, t, fold, "r", ta, tb, M, N, K, al, A, lda, B, ldb, be, C, ldc)


def gpu_gemm(rb, t, fold, ta, tb, M, N, K, A, lda, B, ldb, C, ldc):
    al, be = scalars(t)
    if t == "d":
        rb.call("reproBLAS_rdgemm", fold, "r", ta, tb, M, N, K, al, A, lda, B, ldb, be, C, ldc)
    else:
        rb_gemm(rb, t, fold, "r", ta, tb, M, N, K, al, A, lda, B, ldb, be, C, ldc)


def check_gemm(cuda, rb, port, t, fold, ta, tb, M, N, K, A, B, seed):
    C = ops(t, M * N, seed + 2)
    want = C.copy()
    lda, ldb = (K if ta == "n" else M), (N if tb == "n" else K)
    oracle_gemm(port, t, fold, ta, tb, M, N, K, A, lda, B, ldb, want, N)
    Cd = dev(cuda, C)
    gpu_gemm(rb, t, fold, ta, tb, M, N, K, dev(cuda, A), lda, dev(cuda, B), ldb, Cd, N)
    got = Cd.cpu().numpy().view(FULL[t])
    assert same_value(got.view(REAL[t]), want.view(REAL[t])), (t, fold, ta, tb, M, N, K)


@pytest.mark.parametrize("t", list("dszc"))
@pytest.mark.parametrize("fold", [2, 3, 5, 8])
def test_gemm_cut_tiles(cuda, rb, port, t, fold):
    # few tiles and a long sum: every tile is cut into many parts; then K one beyond, at and
    # before the end of a K block, and sizes one off the tiles
    for i, (M, N, K, ta, tb) in enumerate([(33, 17, 4001, "t", "n"), (1, 1, 3000, "n", "t"), (16, 31, 2047, "n", "n"),
                                           (65, 33, 32, "t", "t"), (32, 64, 33, "n", "n"), (31, 63, 31, "n", "t")]):
        check_gemm(cuda, rb, port, t, fold, ta, tb, M, N, K, ops(t, M * K, i), ops(t, K * N, i + 50), i)


@pytest.mark.parametrize("t", list("dszc"))
def test_gemm_without_scratch(cuda, rb, port, t):
    M, N, K = 33, 17, 4001
    A, B, C = ops(t, M * K, 1), ops(t, K * N, 2), ops(t, M * N, 3)
    want = C.copy()
    oracle_gemm(port, t, 3, "n", "n", M, N, K, A, K, B, N, want, N)
    stream = cuda.cuda.Stream()
    rb.lib.rb_set_stream(stream.cuda_stream)
    try:
        x = cuda.ones(16, dtype=cuda.float64, device="cuda")
        cuda.cuda.synchronize()
        rb.call("reproBLAS_rdsum", 3, 16, x, 1)       # makes the stream's workspace
        rb.lib.rb_debug_fail_allocations(8)           # neither scratch nor tickets can be had
        Ad, Bd, Cd = dev(cuda, A), dev(cuda, B), dev(cuda, C)
        cuda.cuda.synchronize()
        gpu_gemm(rb, t, 3, "n", "n", M, N, K, Ad, K, Bd, N, Cd, N)
        stream.synchronize()
        assert same_bits(Cd.cpu().numpy(), want.view(REAL[t]))
    finally:
        rb.lib.rb_debug_fail_allocations(0)
        rb.lib.rb_set_stream(None)


@pytest.mark.parametrize("t", list("dszc"))
@pytest.mark.parametrize("ta", ["n", "t"])
def test_gemv_without_scratch(cuda, rb, port, t, ta):
    # units that would be cut between CTAs stay whole when their scratch cannot be had
    M, N, al, be = (9000, 700, *scalars(t)) if ta == "n" else (3000, 1500, *scalars(t))
    A, x, y = ops(t, M * N, 1), ops(t, max(M, N), 2), ops(t, M if ta == "n" else N, 3)
    want = y.copy()
    Ad, xd, yd = dev(cuda, A), dev(cuda, x), dev(cuda, y)
    stream = cuda.cuda.Stream()
    rb.lib.rb_set_stream(stream.cuda_stream)
    try:
        one = cuda.ones(16, dtype=cuda.float64, device="cuda")
        cuda.cuda.synchronize()
        rb.call("reproBLAS_rdsum", 3, 16, one, 1)     # makes the stream's workspace
        rb.lib.rb_debug_fail_allocations(8)
        if t == "d":
            port.rdgemv(3, b"r", ta.encode(), M, N, al, ptr(A), N, ptr(x), 1, be, ptr(want), 1)
            rb.call("reproBLAS_rdgemv", 3, "r", ta, M, N, al, Ad, N, xd, 1, be, yd, 1)
        else:
            lib_gemv(port, t, 3, "r", ta, M, N, al, A, N, x, 1, be, want, 1)
            rb_gemv(rb, t, 3, "r", ta, M, N, al, Ad, N, xd, 1, be, yd, 1)
        stream.synchronize()
        assert same_bits(yd.cpu().numpy(), want.view(REAL[t]))
    finally:
        rb.lib.rb_debug_fail_allocations(0)
        rb.lib.rb_set_stream(None)


def test_error_of_an_earlier_call_is_kept(cuda, rb):
    # calls that do without scratch they could not have leave the thread's unread error alone
    Ad, xd, yd = (cuda.ones(n, dtype=cuda.float64, device="cuda") for n in (3000 * 1500, 3000, 3000))
    stream = cuda.cuda.Stream(priority=-1)
    cuda.cuda.synchronize()
    rb.lib.rb_set_stream(stream.cuda_stream)
    try:
        rb.call("reproBLAS_rdsum", 3, 16, Ad, 1)
        rb.lib.reproBLAS_rdsum(1, 16, Ad.data_ptr(), 1)   # fold 1: refused
        code, text = rb.lib.rb_get_last_error(), rb.lib.rb_get_last_error_message()
        assert code != 0
        for fails in (1, 2):
            rb.lib.rb_debug_fail_allocations(fails)
            rb.lib.reproBLAS_rdgemv(3, b"r", b"t", 3000, 1500, 1.5, Ad.data_ptr(), 1500, xd.data_ptr(), 1, 0.0,
                                    yd.data_ptr(), 1)
            rb.lib.rb_debug_fail_allocations(fails)
            rb.lib.reproBLAS_rdgemm(3, b"r", b"n", b"n", 33, 17, 4001, 1.5, Ad.data_ptr(), 4001, Ad.data_ptr(), 17,
                                    0.0, yd.data_ptr(), 17)
            assert (rb.lib.rb_get_last_error(), rb.lib.rb_get_last_error_message()) == (code, text)
        stream.synchronize()
        assert bool((yd[:33 * 17] == 1.5 * 4001).all())
    finally:
        rb.lib.rb_debug_fail_allocations(0)
        rb.lib.rb_clear_error()
        rb.lib.rb_set_stream(None)


@pytest.mark.parametrize("t, ta, M, N", [("d", "n", 20_000_000, 4), ("z", "n", 4_000_000, 8), ("s", "t", 16, 8_000_000),
                                         ("c", "n", 400_003, 100), ("z", "t", 300, 200_000)])
def test_gemv_scratch_does_not_grow_with_the_outputs(cuda, rb, t, ta, M, N):
    # at most two units per CTA are cut: the device memory a call takes stays below 64 MB
    A = cuda.zeros(M * N * (2 if t in "zc" else 1), dtype={"d": cuda.float64, "z": cuda.float64}.get(t, cuda.float32),
                   device="cuda")
    x, y = cuda.zeros_like(A[:2 * max(M, N)]), cuda.ones_like(A[:2 * max(M, N)])
    stream = cuda.cuda.Stream(priority=-1)
    cuda.cuda.synchronize()
    rb.lib.rb_set_stream(stream.cuda_stream)
    try:
        free = cuda.cuda.mem_get_info()[0]
        if t == "d":
            rb.call("reproBLAS_rdgemv", 3, "r", ta, M, N, 1.5, A, N, x, 1, 0.0, y, 1)
        else:
            rb_gemv(rb, t, 3, "r", ta, M, N, 1.5, A, N, x, 1, 0.0, y, 1)
        assert rb.lib.rb_synchronize() == 0
        assert free - cuda.cuda.mem_get_info()[0] < 64 << 20
        n = (M if ta == "n" else N) * (2 if t in "zc" else 1)
        assert int(cuda.count_nonzero(y[:n])) == 0
    finally:
        rb.lib.rb_set_stream(None)


@pytest.mark.parametrize("t", list("dszc"))
def test_gemm_captured(cuda, rb, port, t):
    # a graph must not hold scratch that a later, larger call replaces: capture, grow, replay
    M, N, K = 33, 17, 2000
    A, B, C = ops(t, M * K, 4), ops(t, K * N, 5), ops(t, M * N, 6)
    want = C.copy()
    oracle_gemm(port, t, 3, "n", "n", M, N, K, A, K, B, N, want, N)
    Ad, Bd, Cd = dev(cuda, A), dev(cuda, B), dev(cuda, C)
    big = 400
    Ab, Bb, Cb = dev(cuda, ops(t, big * 5000, 7)), dev(cuda, ops(t, 5000 * big, 8)), dev(cuda, ops(t, big * big, 9))
    graph, stream = cuda.cuda.CUDAGraph(), cuda.cuda.Stream()
    rb.lib.rb_set_stream(stream.cuda_stream)
    try:
        stream.wait_stream(cuda.cuda.current_stream())
        keep = Cd.clone()
        gpu_gemm(rb, t, 3, "n", "n", M, N, K, Ad, K, Bd, N, keep, N)
        stream.synchronize()
        with cuda.cuda.graph(graph, stream=stream):
            gpu_gemm(rb, t, 3, "n", "n", M, N, K, Ad, K, Bd, N, Cd, N)
        gpu_gemm(rb, t, 3, "n", "n", big, big, 5000, Ab, 5000, Bb, big, Cb, big)
        stream.synchronize()
        graph.replay()
        cuda.cuda.synchronize()
        assert same_bits(Cd.cpu().numpy(), want.view(REAL[t]))
    finally:
        rb.lib.rb_set_stream(None)


def test_first_calls_on_a_stream_while_the_default_stream_is_busy(cuda, rb, port):
    # a new workspace's tickets and status word must be zero before its non-blocking stream uses
    # them, whatever is queued on the legacy default stream: products cut between CTAs are the
    # stream's first calls here, behind no work of their own
    M, N, K = 33, 17, 4001
    A, B, C = ops("d", M * K, 1), ops("d", K * N, 2), ops("d", M * N, 3)
    want = C.copy()
    oracle_gemm(port, "d", 3, "n", "n", M, N, K, A, K, B, N, want, N)
    m, n = 9000, 700
    G, x, y = ops("d", m * n, 4), ops("d", n, 5), ops("d", m, 6)
    wy = y.copy()
    port.rdgemv(3, b"r", b"n", m, n, 1.5, ptr(G), n, ptr(x), 1, 0.5, ptr(wy), 1)
    Ad, Bd, Cd, Gd, xd, yd = (dev(cuda, v) for v in (A, B, C, G, x, y))
    big = cuda.rand(8192, 8192, device="cuda")
    for first in ("gemm", "gemv"):
        stream = cuda.cuda.Stream(priority=-1)   # a pool of its own: no call has used its streams
        cuda.cuda.synchronize()
        for _ in range(20):
            big @ big
        rb.lib.rb_set_stream(stream.cuda_stream)
        try:
            if first == "gemm":
                gpu_gemm(rb, "d", 3, "n", "n", M, N, K, Ad, K, Bd, N, Cd, N)
            else:
                rb.call("reproBLAS_rdgemv", 3, "r", "n", m, n, 1.5, Gd, n, xd, 1, 0.5, yd, 1)
            assert rb.lib.rb_synchronize() == 0
        finally:
            rb.lib.rb_set_stream(None)
        cuda.cuda.synchronize()
    assert same_bits(Cd.cpu().numpy(), want)
    assert same_bits(yd.cpu().numpy(), wy)


def test_batch_plan_made_while_the_default_stream_is_busy(cuda, rb):
    from test_batched_gpu import Problem
    big, stream = cuda.rand(8192, 8192, device="cuda"), cuda.cuda.Stream(priority=-1)
    P = Problem(cuda, rb, nseg=200, max_log2=16, ngemm=8, seed=3)
    try:
        want, want_c = P.expected_segments()[0], P.expected_gemms()
        cuda.cuda.synchronize()
        for _ in range(20):
            big @ big
        assert rb.call("rb_batch_plan_set_config", P.plan, 1, 1 << 13, 512, 0) == 0
        assert rb.call("rb_batch_plan_run", P.plan, stream.cuda_stream) == 0
        cuda.cuda.synchronize()
        assert same_bits(P.results.cpu().numpy(), want)
        for got, w in zip(P.gemm_outputs(), want_c):
            assert same_bits(got, w)
    finally:
        P.destroy()


@pytest.mark.parametrize("t", list("dszc"))
@pytest.mark.parametrize("ta", ["n", "t"])
def test_gemv_captured(cuda, rb, port, t, ta):
    # the same for gemv, through the streaming and the direct kernels
    M, N, al, be = 3000, 1500, *scalars(t)
    A, x, y = ops(t, M * N, 4), ops(t, max(M, N), 5), ops(t, max(M, N), 6)
    want = y.copy()
    if t == "d":
        port.rdgemv(3, b"r", ta.encode(), M, N, al, ptr(A), N, ptr(x), 1, be, ptr(want), 1)
    else:
        lib_gemv(port, t, 3, "r", ta, M, N, al, A, N, x, 1, be, want, 1)
    Ad, xd, yd, keep = dev(cuda, A), dev(cuda, x), dev(cuda, y), dev(cuda, y)
    rows = 9000
    Ab, xb, yb = dev(cuda, ops(t, rows * N, 7)), dev(cuda, ops(t, rows, 8)), dev(cuda, ops(t, rows, 9))

    def call(m, a, v, out):
        if t == "d":
            rb.call("reproBLAS_rdgemv", 3, "r", ta, m, N, al, a, N, v, 1, be, out, 1)
        else:
            rb_gemv(rb, t, 3, "r", ta, m, N, al, a, N, v, 1, be, out, 1)

    graph, stream = cuda.cuda.CUDAGraph(), cuda.cuda.Stream()
    rb.lib.rb_set_stream(stream.cuda_stream)
    try:
        stream.wait_stream(cuda.cuda.current_stream())
        call(M, Ad, xd, keep)
        stream.synchronize()
        with cuda.cuda.graph(graph, stream=stream):
            call(M, Ad, xd, yd)
        call(rows, Ab, xb, yb)
        stream.synchronize()
        graph.replay()
        cuda.cuda.synchronize()
        assert same_bits(yd.cpu().numpy(), want.view(REAL[t]))
    finally:
        rb.lib.rb_set_stream(None)


@pytest.mark.parametrize("t, ta, M, N", [("d", "n", 100, 60000), ("d", "t", 3000, 1500), ("s", "t", 40000, 100),
                                         ("z", "n", 3000, 1500), ("z", "t", 2000, 500), ("c", "n", 9000, 300)])
def test_gemv_replays_beside_other_calls(cuda, rb, port, t, ta, M, N):
    # a captured call whose units are cut has scratch of its own: captured with the workspace warmed by
    # a reduction alone, replayed on one stream while the stream it was captured on runs other
    # calls; a second graph of the same call at the same time; and after the graphs are gone
    al, be = scalars(t)
    A, x, y = ops(t, M * N, 4), ops(t, max(M, N), 5), ops(t, M if ta == "n" else N, 6)
    want = y.copy()
    if t == "d":
        port.rdgemv(3, b"r", ta.encode(), M, N, al, ptr(A), N, ptr(x), 1, be, ptr(want), 1)
    else:
        lib_gemv(port, t, 3, "r", ta, M, N, al, A, N, x, 1, be, want, 1)
    Ad, xd, y0 = dev(cuda, A), dev(cuda, x), dev(cuda, y)

    def call(out):
        if t == "d":
            rb.call("reproBLAS_rdgemv", 3, "r", ta, M, N, al, Ad, N, xd, 1, be, out, 1)
        else:
            rb_gemv(rb, t, 3, "r", ta, M, N, al, Ad, N, xd, 1, be, out, 1)

    stream, others = cuda.cuda.Stream(priority=-1), [cuda.cuda.Stream(), cuda.cuda.Stream()]
    rb.lib.rb_set_stream(stream.cuda_stream)
    try:
        one = cuda.ones(16, dtype=cuda.float64, device="cuda")
        cuda.cuda.synchronize()
        rb.call("reproBLAS_rdsum", 3, 16, one, 1)
        for again in range(2):
            outs = [y0.clone() for _ in range(3)]
            cuda.cuda.synchronize()
            graphs = []
            for k in range(2):
                g = cuda.cuda.CUDAGraph()
                with cuda.cuda.graph(g, stream=stream):
                    outs[k].copy_(y0)
                    call(outs[k])
                graphs.append(g)
            for rep in range(20):
                for k in range(2):
                    with cuda.cuda.stream(others[k]):
                        graphs[k].replay()
                with cuda.cuda.stream(stream):
                    outs[2].copy_(y0)
                call(outs[2])
            cuda.cuda.synchronize()
            for out in outs:
                assert same_bits(out.cpu().numpy(), want.view(REAL[t])), again
            del graphs, g
    finally:
        rb.lib.rb_set_stream(None)


@pytest.mark.parametrize("t", list("dszc"))
@pytest.mark.parametrize("fold", [2, 3, 4])
def test_gemm_blocks_off_the_unchecked_path(cuda, rb, port, t, fold):
    M, N, K = 40, 35, 100
    A, B = ops(t, M * K, 11).reshape(M, K), ops(t, K * N, 12).reshape(K, N)
    hi, lo = (2.0 ** 500, 2.0 ** -500) if t in "dz" else (2.0 ** 60, 2.0 ** -60)
    A[0] = 0                        # a zero row
    A[1] *= lo                      # the finest bins (products down to the subnormals)
    B[:, 2] *= lo
    A[2, 70] *= hi                  # a raise in the third K block
    A[3] *= hi                      # products near the top: the compressed first bin
    B[:, 3] *= hi
    check_gemm(cuda, rb, port, t, fold, "n", "n", M, N, K, A.ravel(), B.ravel(), 13)
    A[4, 5], A[5, 90], A[6, 0] = np.inf, -np.inf, np.nan
    A[7, 1], A[7, 2] = np.inf, -np.inf
    C = ops(t, M * N, 15)
    want = C.copy()
    oracle_gemm(port, t, fold, "n", "n", M, N, K, A.ravel(), K, B.ravel(), N, want, N)
    Cd = dev(cuda, C)
    gpu_gemm(rb, t, fold, "n", "n", M, N, K, dev(cuda, A.ravel()), K, dev(cuda, B.ravel()), N, Cd, N)
    assert same_value(Cd.cpu().numpy(), want.view(REAL[t]))


@pytest.mark.parametrize("t", list("dszc"))
@pytest.mark.parametrize("fold", [2, 3, 7, 8])
def test_gemm_short_sums(cuda, rb, port, t, fold):
    # sums shorter than a K block, whose entries all take their index from the largest of few products:
    # magnitudes around the borders between indices, and FP64 products of 2^1017 and more, whose high
    # words are a float's NaN; beta 0 reads no C
    for i, (M, N, K) in enumerate([(33, 65, 1), (70, 40, 2), (31, 33, 5), (64, 64, 8), (40, 70, 33)]):
        A, B = ops(t, M * K, i).reshape(M, K), ops(t, K * N, i + 50).reshape(K, N)
        e = (np.arange(M) - M // 2) * (24 if t in "dz" else 3)
        A *= np.exp2(np.clip(e, -500, 510) if t in "dz" else np.clip(e, -60, 62)).astype(REAL[t])[:, None]
        check_gemm(cuda, rb, port, t, fold, "n", "n", M, N, K, A.ravel(), B.ravel(), i)
        B[:, 3:9] *= REAL[t](2.0 ** 511 if t in "dz" else 2.0 ** 62)
        check_gemm(cuda, rb, port, t, fold, "n", "n", M, N, K, A.ravel(), B.ravel(), i)
        al = scalars(t)[0]
        want, C = np.zeros(M * N, FULL[t]), dev(cuda, np.full(M * N, np.nan, FULL[t]))
        Ad, Bd = dev(cuda, A.ravel()), dev(cuda, B.ravel())
        if t == "d":
            port.rdgemm(fold, b"r", b"n", b"n", M, N, K, al, ptr(A), K, ptr(B), N, 0.0, ptr(want), N)
            rb.call("reproBLAS_rdgemm", fold, "r", "n", "n", M, N, K, al, Ad, K, Bd, N, 0.0, C, N)
        else:
            lib_gemm(port, t, fold, "r", "n", "n", M, N, K, al, A, K, B, N, 0.0, want, N)
            rb_gemm(rb, t, fold, "r", "n", "n", M, N, K, al, Ad, K, Bd, N, 0.0, C, N)
        assert same_value(C.cpu().numpy(), want.view(REAL[t])), (t, fold, M, N, K)


def gemv_both(cuda, rb, port, t, fold, ta, M, N, lda, off, incx, seed, dist="normal"):
    """A starting `off` reals into its buffer, against the oracle"""
    al, be = scalars(t)
    per = 1 if t in "ds" else 2
    buf = gen(dist, off + M * lda * per, seed, REAL[t])
    A = np.ascontiguousarray(buf[off:]).view(FULL[t])
    nx, ny = (N, M) if ta == "n" else (M, N)
    x, y = ops(t, nx * incx, seed + 1, dist), ops(t, ny, seed + 2, dist)
    want = y.copy()
    Ad = cuda.from_numpy(buf).cuda()[off:]
    yd = dev(cuda, y)
    if t == "d":
        port.rdgemv(fold, b"r", ta.encode(), M, N, al, ptr(A), lda, ptr(x), incx, be, ptr(want), 1)
        rb.call("reproBLAS_rdgemv", fold, "r", ta, M, N, al, Ad, lda, dev(cuda, x), incx, be, yd, 1)
    else:
        lib_gemv(port, t, fold, "r", ta, M, N, al, A, lda, x, incx, be, want, 1)
        rb_gemv(rb, t, fold, "r", ta, M, N, al, Ad, lda, dev(cuda, x), incx, be, yd, 1)
    assert rb.lib.rb_synchronize() == 0
    assert same_bits(yd.cpu().numpy(), want.view(REAL[t])), (t, fold, ta, M, N, lda, off, incx)


@pytest.mark.parametrize("t", list("dszc"))
@pytest.mark.parametrize("ta", ["n", "t"])
def test_gemv_alignments(cuda, rb, port, t, ta):
    # above the direct kernels' limits, so that the streaming kernel takes the rows in 1, 2 and 4
    # phases: every distance of A from a 16-byte boundary, leading dimensions of all residues
    M, N = (8200, 130) if ta == "n" else (3000, 1500)
    for off in range(4):
        for pad in range(4):
            gemv_both(cuda, rb, port, t, 3, ta, M, N, N + pad, off, 1 + (off & 1), 31 * off + pad)


@pytest.mark.parametrize("t", list("dszc"))
@pytest.mark.parametrize("fold", [2, 4, 6, 8])
def test_gemv_stream_folds(cuda, rb, port, t, fold):
    for ta, M, N, pad in [("n", 8193, 257, 1), ("t", 255, 9000, 1), ("t", 2049, 2050, 0), ("n", 8200, 64, 0)]:
        gemv_both(cuda, rb, port, t, fold, ta, M, N, N + pad, 0, 1, fold)


@pytest.mark.parametrize("fold, ta", [(2, "t"), (3, "c"), (4, "t"), (6, "c"), (7, "t")])
def test_gemv_large_complex_columns(cuda, rb, port, fold, ta):
    # FP64 complex columns above 192 MB: the streaming kernel up to fold 6
    for M, N in [(41003, 307), (307, 41003)]:
        gemv_both(cuda, rb, port, "z", fold, ta, M, N, N + 1, 0, 1, fold)


@pytest.mark.parametrize("t", list("dszc"))
@pytest.mark.parametrize("fold", [2, 3, 8])
def test_gemv_few_long_rows(cuda, rb, port, t, fold):
    # rows cut between CTAs: around the first cut (seven steps of 8 warps), ragged last parts, both
    # sides of the limits of 24 and 48 rows, every alignment, strided x, units that all CTAs share
    # (their parts summed in two stages), and raises and non-finite values in a late part
    step = 1024
    for i, (M, N) in enumerate([(1, 7 * step - 1), (1, 7 * step), (2, 8 * step + 1), (3, 100003), (24, 9001), (25, 9003),
                                (48, 70001), (49, 70003), (64, 90001), (1, 600011)]):
        gemv_both(cuda, rb, port, t, fold, "n", M, N, N + (i & 3), i & 3, 1 + (i & 1), i)
    M, N = 2, 200000
    al, be = scalars(t)
    A = ops(t, M * N, 5).reshape(M, N)
    A[0, N - 5] = 2.0 ** (600 if t in "dz" else 90)
    A[1, 150000], A[1, 7] = np.inf, 2.0 ** (1000 if t in "dz" else 120)
    x, y = ops(t, N, 6), ops(t, M, 7)
    want = y.copy()
    yd = dev(cuda, y)
    if t == "d":
        port.rdgemv(fold, b"r", b"n", M, N, al, ptr(A), N, ptr(x), 1, be, ptr(want), 1)
        rb.call("reproBLAS_rdgemv", fold, "r", "n", M, N, al, dev(cuda, A.ravel()), N, dev(cuda, x), 1, be, yd, 1)
    else:
        lib_gemv(port, t, fold, "r", "n", M, N, al, A, N, x, 1, be, want, 1)
        rb_gemv(rb, t, fold, "r", "n", M, N, al, dev(cuda, A.ravel()), N, dev(cuda, x), 1, be, yd, 1)
    assert same_value(yd.cpu().numpy(), want.view(REAL[t]))


@pytest.mark.parametrize("fold", [5, 6, 7, 8])
def test_gemv_complex_rows_of_high_folds(cuda, rb, port, fold):
    # FP64 complex rows from fold 6 on take the direct kernel from 500 elements a row
    for i, (M, N) in enumerate([(6200, 499), (6200, 500), (700, 5003)]):
        gemv_both(cuda, rb, port, "z", fold, "n", M, N, N + i, i & 1, 1, fold)


@pytest.mark.parametrize("t", list("dszc"))
@pytest.mark.parametrize("ta", ["n", "t"])
def test_gemv_without_products(cuda, rb, port, t, ta):
    # alpha 0 deposits nothing, whatever A and x hold: y is beta*y
    for M, N in [(9001, 70), (70, 9001), (300, 300), (3000, 3001)]:
        A, y = ops(t, M * N, 1), ops(t, M if ta == "n" else N, 2)
        A[3] = np.nan
        x = np.full(max(M, N), np.inf, FULL[t])
        be, want = scalars(t)[1], y.copy()
        al = 0.0 if t in "ds" else 0j
        yd = dev(cuda, y)
        if t == "d":
            port.rdgemv(3, b"r", ta.encode(), M, N, al, ptr(A), N, ptr(x), 1, be, ptr(want), 1)
            rb.call("reproBLAS_rdgemv", 3, "r", ta, M, N, al, dev(cuda, A), N, dev(cuda, x), 1, be, yd, 1)
        else:
            lib_gemv(port, t, 3, "r", ta, M, N, al, A, N, x, 1, be, want, 1)
            rb_gemv(rb, t, 3, "r", ta, M, N, al, dev(cuda, A), N, dev(cuda, x), 1, be, yd, 1)
        assert same_bits(yd.cpu().numpy(), want.view(REAL[t])), (M, N)


@pytest.mark.parametrize("t", list("dszc"))
@pytest.mark.parametrize("fold", [2, 3, 6])
def test_gemv_short_columns(cuda, rb, port, t, fold):
    # many columns of few rows: both sides of the limits on each, whole and partial steps of four rows
    most = {"d": 128, "s": 48, "z": 384, "c": 128}[t]
    for i, (M, N) in enumerate([(1, 80001), (3, 80000), (5, 79999), (8, 100003), (most, 80000), (most + 1, 80001)]):
        gemv_both(cuda, rb, port, t, fold, "t", M, N, N + (i & 3), i & 3, 1 + (i & 1), i)


@pytest.mark.parametrize("t", list("dszc"))
@pytest.mark.parametrize("ta", ["n", "t"])
def test_gemv_few_rows_and_limits(cuda, rb, port, t, ta):
    es = {"d": 8, "s": 4, "z": 16, "c": 8}[t]
    rows = 300
    limit = (24 if ta == "n" else 16) << 20
    n = limit // (rows * es)
    shapes = [(1, 70001), (2, 9001), (3, 4097), (rows, n), (rows, n + 1), (255, 300), (256, 300), (8192, 5), (8193, 5)]
    for i, (M, N) in enumerate(shapes):
        gemv_both(cuda, rb, port, t, 3, ta, M, N, N + (i & 1), 0, 1, i)
    # infinities, NaN and the top bin through the streaming kernel
    M, N = (8200, 64) if ta == "n" else (200, 8200)
    al, be = scalars(t)
    A = ops(t, M * N, 5).reshape(M, N)
    A[5, 3], A[6, 4], A[7, 5] = np.inf, np.nan, -np.inf
    A[9] *= 2.0 ** (1000 if t in "dz" else 120)
    x, y = ops(t, N if ta == "n" else M, 6), ops(t, M if ta == "n" else N, 7)
    want = y.copy()
    yd = dev(cuda, y)
    if t == "d":
        port.rdgemv(3, b"r", ta.encode(), M, N, al, ptr(A), N, ptr(x), 1, be, ptr(want), 1)
        rb.call("reproBLAS_rdgemv", 3, "r", ta, M, N, al, dev(cuda, A.ravel()), N, dev(cuda, x), 1, be, yd, 1)
    else:
        lib_gemv(port, t, 3, "r", ta, M, N, al, A, N, x, 1, be, want, 1)
        rb_gemv(rb, t, 3, "r", ta, M, N, al, dev(cuda, A.ravel()), N, dev(cuda, x), 1, be, yd, 1)
    assert same_value(yd.cpu().numpy(), want.view(REAL[t]))


@pytest.mark.parametrize("fold", [2, 3, 4])
def test_sums_of_squares_scales(cuda, rb, port, fold):
    # the scale grows element by element, lane by lane and warp by warp, across the steps of the
    # scale (40 binades, 13 in FP32) and around 1; non-finite values at a tile's ends
    for dt, names, lo, hi in [(np.float64, ("dbdssq", "rdnrm2"), -120, 120), (np.float32, ("sbsssq", "rsnrm2"), -50, 50)]:
        for n in (1, 15, 512, 4099, 70001):
            e = np.linspace(lo, hi, n)
            for k, ex in enumerate((e, e[::-1], np.round(e / 13) * 13, np.where(np.arange(n) % 64 < 32, lo, hi))):
                x = np.exp2(np.asarray(ex, dtype=np.float64)).astype(dt)
                x[1::2] *= dt(-1.25)
                X = cuda.from_numpy(x).cuda()
                want = binned_zeros(fold, "d" if dt is np.float64 else "s")
                ws = getattr(port, names[0])(fold, n, ptr(x), 1, 0.0, ptr(want))
                Z = cuda.zeros(2 * fold, dtype=X.dtype, device="cuda")
                gs = rb.call("binnedBLAS_" + names[0], fold, n, X, 1, 0.0, Z)
                assert gs == ws, (dt, n, k)
                assert same_state(Z.cpu().numpy(), want, fold, 1), (dt, n, k)
                assert rb.call("reproBLAS_" + names[1], fold, n, X, 1) == getattr(port, names[1])(fold, n, ptr(x), 1)
            for bad in (np.inf, -np.inf, np.nan):
                y = x.copy()
                y[-1] = bad
                a = rb.call("reproBLAS_" + names[1], fold, n, cuda.from_numpy(y).cuda(), 1)
                b = getattr(port, names[1])(fold, n, ptr(y), 1)
                assert a == b or (a != a and b != b)


@pytest.mark.parametrize("S", [2, 5, 8, 12])
def test_int8_digits_of_small_magnitudes(cuda, rb, S):
    # elements up to 2^200 below their row's largest (their digits lie behind the last slice),
    # subnormals, zero rows and columns: the digits of r <- 128 r, d <- trunc(r), r <- r - d
    rng = np.random.default_rng(S)
    M, N, K = 70, 65, 90
    A = np.ldexp(rng.uniform(1, 2, (M, K)), rng.integers(-200, 1, (M, K))) * rng.choice([-1.0, 1.0], (M, K))
    B = np.ldexp(rng.uniform(1, 2, (K, N)), rng.integers(-90, 1, (K, N))) * rng.choice([-1.0, 1.0], (K, N))
    A[3] = 0
    B[:, 4] = 0
    A[5] = 5e-324 * rng.integers(-9, 10, K)
    Mp, Np, Kp = -(-M // 128) * 128, -(-N // (64 if S <= 4 else 32)) * (64 if S <= 4 else 32), -(-K // 32) * 32
    z = lambda n, t: cuda.zeros(n, dtype=t, device="cuda")
    raw, As, Bs = z(S * Mp * Np, cuda.int32), z(S * Mp * Kp, cuda.int8), z(S * Np * Kp, cuda.int8)
    ea, fb = z(M, cuda.int32), z(N, cuda.int32)
    assert rb.call("rb_dgemm_int8_inspect", M, N, K, cuda.from_numpy(A).cuda(), cuda.from_numpy(B).cuda(), S, raw,
                   As, Bs, ea, fb) == 0
    for X, dig, ex, R, Rp in [(A, As, ea, M, Mp), (B.T, Bs, fb, N, Np)]:
        e = np.frexp(np.abs(X).max(axis=1))[1]
        assert np.array_equal(ex.cpu().numpy(), e)
        d = dig.cpu().numpy().reshape(Kp // 16, S, Rp // 8, 8, 16).transpose(1, 2, 3, 0, 4).reshape(S, Rp, Kp)
        r = np.ldexp(X, -e[:, None])
        for p in range(S):
            r = r * 128
            t = np.trunc(r)
            r = r - t
            assert np.array_equal(d[p, :R, :K], t.astype(np.int8)), p
        assert not d[:, R:].any() and not d[:, :, K:].any()


@pytest.mark.parametrize("ta", ["n", "t", "c"])
def test_gemv_rows_of_more_than_16_gib(cuda, rb, port, ta):
    # FP64 complex rows of more than 2^30 elements (2^31 words of 8 bytes): products on both sides
    # of element 2^30 count. The matrix is zero but for a few elements and x has stride 0 (one
    # element), so the oracle's sum is that of the few
    n = 2 ** 30 + 300
    at = [0, 5, 2 ** 30 - 1, 2 ** 30, 2 ** 30 + 1, n - 1]
    vals, x = ops("z", len(at), 3), ops("z", 1, 4)
    al, be = 1.5 - 0.25j, 0.0
    A = cuda.zeros((n, 2), dtype=cuda.float64, device="cuda")
    A[cuda.tensor(at, device="cuda")] = cuda.from_numpy(vals.view(np.float64).reshape(-1, 2)).cuda()
    if ta == "n":
        # row-major, one row; column-major, the transpose of one column
        want = np.zeros(1, np.complex128)
        lib_gemv(port, "z", 3, "r", "n", 1, len(at), al, vals, len(at), x, 0, be, want, 1)
        for order, t, M, N, lda in [("r", "n", 1, n, n), ("c", "t", n, 1, n)]:
            y = dev(cuda, np.zeros(1, np.complex128))
            rb_gemv(rb, "z", 3, order, t, M, N, al, A, lda, dev(cuda, x), 0, be, y, 1)
            assert same_bits(y.cpu().numpy(), want.view(np.float64)), order
        return
    # one row, transposed: n outputs of one product each
    want = np.zeros(len(at), np.complex128)
    lib_gemv(port, "z", 3, "r", ta, 1, len(at), al, vals, len(at), x, 0, be, want, 1)
    y = cuda.full((n, 2), 7.0, dtype=cuda.float64, device="cuda")
    rb_gemv(rb, "z", 3, "r", ta, 1, n, al, A, n, dev(cuda, x), 0, be, y, 1)
    got = y[cuda.tensor(at, device="cuda")].cpu().numpy()
    assert same_bits(got.ravel(), want.view(np.float64))
    assert int(cuda.count_nonzero(y)) == np.count_nonzero(want.view(np.float64))


@pytest.mark.parametrize("t", list("dszc"))
@pytest.mark.parametrize("fold", [2, 3, 6])
def test_gemv_streams_as_built(cuda, rb, t, fold):
    # the streaming kernels run, not the direct ones that stand in where the compiler gave FP64 complex
    # other registers than the kernel deals out: only a pipeline can be told to stop feeding its ring
    n = 4096
    A, x, y = (cuda.ones(k * 2, dtype=cuda.float64 if t in "dz" else cuda.float32, device="cuda")
               for k in (n * n, n, n))
    lib = rb.lib
    for ta in "t" if t == "z" and fold == 6 else "nt":   # (FP64 complex rows of fold 6 go direct)
        try:
            lib.rb_clear_error()
            lib.rb_debug_pipeline_fault(2, 20000)
            if t == "d":
                rb.call("reproBLAS_rdgemv", fold, "r", ta, n, n, 1.5, A, n, x, 1, 0.0, y, 1)
            else:
                rb_gemv(rb, t, fold, "r", ta, n, n, 1.5, A, n, x, 1, 0.0, y, 1)
            assert lib.rb_synchronize() == 2 and b"timed out" in lib.rb_get_last_error_message(), ta
        finally:
            lib.rb_debug_pipeline_fault(-1, 0)
            lib.rb_clear_error()
    assert lib.rb_synchronize() == 0

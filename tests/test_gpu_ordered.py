"""Searches over spatially ordered clouds against the sweeping kernels, bit for bit.

Both run through the same C entry point: with a scratch buffer the clouds are ordered, without one
every pair is swept (and the sweeping kernels are compared with the oracle elsewhere).  Sizes sit at
the edges of the structure: leaves of 8 points, windows of 256, clusters of one to eight blocks, several
chunks of 32 windows.  The inputs cover what orders badly: duplicates, a
lattice full of ties, a plane, an outlier that stretches the grid, NaN and infinite coordinates.
All results are decided on exactly rounded distances, so the comparison is exact.
"""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"

KINDS = ("uniform", "lattice", "zeros", "same", "plane", "outlier", "nonfinite", "wide")


def _cloud(kind, B, N, g):
    p = torch.randn(B, N, 3, generator=g)
    if kind == "uniform":
        p = torch.rand(B, N, 3, generator=g)
    elif kind == "lattice":
        p = torch.randint(0, 9, (B, N, 3), generator=g).float() * 0.1
    elif kind == "zeros":
        p[torch.rand(B, N, generator=g) < 0.3] = 0
    elif kind == "same":
        p = torch.full((B, N, 3), 0.25)
    elif kind == "plane":
        p[..., 2] = 1.5
    elif kind == "outlier":
        p[:, N // 2] = 1e6
    elif kind == "nonfinite":
        p[0, 5, 1], p[B - 1, 7, 2] = float("nan"), float("inf")
    elif kind == "wide":
        p = p * 1e18
    return p


def _pair(kind, B, N, M, cf):
    g = torch.Generator().manual_seed(N + M)
    a, b = _cloud(kind, B, N, g), _cloud(kind, B, M, g)
    if cf:
        a, b = a.transpose(1, 2).contiguous(), b.transpose(1, 2).contiguous()
    return a.to(DEV), b.to(DEV)


def _stream():
    return torch.cuda.current_stream().cuda_stream


def _scratch():
    return torch.full((96 << 20,), 0xA5, dtype=torch.uint8, device=DEV)


def _same(x, y):
    return torch.equal(x.view(torch.int32) if x.dtype == torch.float32 else x,
                       y.view(torch.int32) if y.dtype == torch.float32 else y)


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("B,N,M,cf", [(3, 513, 1100, 0), (2, 4097, 1024, 1), (1, 20000, 33000, 0)])
def test_chamfer(kind, B, N, M, cf):
    from torkit3d_b200 import _lib

    lib = _lib.load()
    a, b = _pair(kind, B, N, M, cf)
    res = []
    for buf in (None, _scratch()):
        d1, d2 = torch.empty(B, N, device=DEV), torch.empty(B, M, device=DEV)
        i1, i2 = (torch.empty(B, n, dtype=torch.int64, device=DEV) for n in (N, M))
        sums = torch.empty(2, dtype=torch.float64, device=DEV)
        assert lib.tk3d_chamfer_fwd_ws(a.data_ptr(), b.data_ptr(), B, N, M, cf, d1.data_ptr(), i1.data_ptr(),
                                       d2.data_ptr(), i2.data_ptr(), sums.data_ptr(),
                                       buf.data_ptr() if buf is not None else None,
                                       buf.numel() if buf is not None else 0, _lib.F32, _stream()) == 0
        res.append((d1, i1, d2, i2, sums))
    for x, y in zip(res[0][:4], res[1][:4]):
        assert _same(x, y)
    torch.testing.assert_close(res[0][4], res[1][4], rtol=1e-12, atol=0, equal_nan=True)  # float64 sums, any order


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("k", [1, 2, 3, 4, 5, 16, 17, 32, 33, 64])  # every list size, both ends of each class count
@pytest.mark.parametrize("B,N,M,cf", [(3, 33, 1100, 0), (2, 4097, 1056, 1), (1, 700, 40001, 0)])
def test_knn(kind, k, B, N, M, cf):
    from torkit3d_b200 import _lib

    lib = _lib.load()
    a, b = _pair(kind, B, N, M, cf)
    for itype, code in ((torch.int64, _lib.I64), (torch.int32, _lib.I32)):
        res = []
        for buf in (None, _scratch()):
            d, i = torch.empty(B, N, k, device=DEV), torch.empty(B, N, k, dtype=itype, device=DEV)
            assert lib.tk3d_knn_ws(a.data_ptr(), b.data_ptr(), B, N, M, k, cf, d.data_ptr(), i.data_ptr(), code,
                                   buf.data_ptr() if buf is not None else None,
                                   buf.numel() if buf is not None else 0, _lib.F32, _stream()) == 0
            res.append((d, i))
        assert _same(res[0][0], res[1][0]) and torch.equal(res[0][1], res[1][1])


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("radius", [0.0, 0.03, 0.15, 0.4, 30.0, float("inf"), float("nan")])  # none, sparse, dense, all
@pytest.mark.parametrize("B,N,M,k,cf", [(2, 333, 1100, 8, 0), (2, 1001, 4099, 40, 1), (1, 2000, 33000, 200, 0)])
def test_ball_query(kind, radius, B, N, M, k, cf):
    from torkit3d_b200 import _lib

    lib = _lib.load()
    a, b = _pair(kind, B, N, M, cf)
    for itype, code in ((torch.int64, _lib.I64), (torch.int32, _lib.I32)):
        res = []
        for buf in (None, _scratch()):
            i = torch.full((B, N, k), -7, dtype=itype, device=DEV)
            assert lib.tk3d_ball_query_ws(a.data_ptr(), b.data_ptr(), B, N, M, radius, k, cf, i.data_ptr(), code,
                                          buf.data_ptr() if buf is not None else None,
                                          buf.numel() if buf is not None else 0, _lib.F32, _stream()) == 0
            res.append(i)
        assert torch.equal(res[0], res[1])


@pytest.mark.parametrize("K", [7, 32])
@pytest.mark.parametrize("radius", [0.05, 0.5])
def test_set_abstraction_from_ordered_neighbours(radius, K):
    from torkit3d_b200 import _lib

    lib = _lib.load()
    B, C, N, M = 4, 12, 16400, 2100
    a, b = _pair("uniform", B, M, N, 1)  # centroids, points
    f = torch.randn(B, C, N, device=DEV)
    need, rows = lib.tk3d_sa_group_scratch_bytes(B, C, N, M, K, _lib.F32), B * C * N * 4
    assert need > rows
    for want_index in (True, False):
        res = []
        for n in (rows, need):  # the smaller buffer holds the transposed features only: the kernel sweeps
            buf = torch.zeros(n, dtype=torch.uint8, device=DEV)
            out = torch.empty(B, C + 3, M, K, device=DEV)
            i = torch.full((B, M, K), -7, dtype=torch.int32, device=DEV)
            st = torch.zeros(1, dtype=torch.int32, device=DEV)
            assert lib.tk3d_sa_group_fwd(b.data_ptr(), a.data_ptr(), f.data_ptr(), B, C, N, M, radius, K, 1, 1,
                                         out.data_ptr(), i.data_ptr() if want_index else None, st.data_ptr(),
                                         buf.data_ptr(), n, _lib.F32, _stream()) == 0
            torch.cuda.synchronize()
            res.append((out, i, st))
        assert _same(res[0][0], res[1][0]) and torch.equal(res[0][1], res[1][1]) and torch.equal(res[0][2], res[1][2])


@pytest.mark.parametrize("kind", ["uniform", "nonfinite", "zeros"])
def test_three_nn_weights_of_the_fused_interpolation(kind):
    from torkit3d_b200 import _fused, ops

    B, C, N, M = 2, 8, 9000, 4100
    a, b = _pair(kind, B, N, M, 1)
    f = torch.randn(B, C, M, device=DEV)
    _, index, weight = _fused.three_nn_interp_forward(a, b, f)
    d, i = ops.knn_points(a[:, :, :2000].contiguous(), b, 3, transpose=True)  # too few pairs to be ordered
    assert torch.equal(index[:, :2000].long(), i)
    assert _same(weight[:, :2000].contiguous(), ops.three_nn_weight(d))


def test_a_scratch_buffer_that_is_too_small_sweeps():
    from torkit3d_b200 import _lib

    lib = _lib.load()
    B, N = 2, 8192
    need = lib.tk3d_knn_scratch_bytes(B, N, N, 3, _lib.F32)
    assert need > 0 and lib.tk3d_knn_scratch_bytes(B, N, N, 3, _lib.F64) == 0
    assert lib.tk3d_knn_scratch_bytes(1, 64, 512, 3, _lib.F32) == 0  # too small to pay
    a, b = _pair("uniform", B, N, N, 0)
    buf, res = torch.zeros(need, dtype=torch.uint8, device=DEV), []
    for n in (need - 1, need):
        d, i = torch.empty(B, N, 3, device=DEV), torch.empty(B, N, 3, dtype=torch.int64, device=DEV)
        assert lib.tk3d_knn_ws(a.data_ptr(), b.data_ptr(), B, N, N, 3, 0, d.data_ptr(), i.data_ptr(), _lib.I64,
                               buf.data_ptr(), n, _lib.F32, _stream()) == 0
        torch.cuda.synchronize()
        assert bool(buf.any()) == (n == need)
        res.append((d, i))
    assert _same(res[0][0], res[1][0]) and torch.equal(res[0][1], res[1][1])


def test_ordered_searches_are_captured_and_replayed_on_new_inputs():
    from torkit3d_b200 import ops

    a, b = _pair("uniform", 2, 9000, 9000, 0)

    def run():
        return ops.nn_distance(a, b) + list(ops.knn_points(a, b, 3)) + list(ops.knn_points(a, b, 20)) + [
            ops.ball_query(a, b, 0.05, 16, transpose=False)]

    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        run()
    torch.cuda.current_stream().wait_stream(s)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = run()
    for kind in ("plane", "outlier"):
        a2, b2 = _pair(kind, 2, 9000, 9000, 0)
        a.copy_(a2), b.copy_(b2)
        graph.replay()
        torch.cuda.synchronize()
        for x, y in zip(out, run()):
            assert _same(x, y)


def test_batches_beyond_the_scratch_limit_are_cut():
    from torkit3d_b200 import _lib

    lib = _lib.load()
    B, N = 9001, 1024  # about 670 MB of index: built in two parts
    g = torch.Generator(device=DEV).manual_seed(1)
    a, b = (torch.randn(B, N, 3, generator=g, device=DEV) for _ in range(2))
    a[4000, 3, 1] = float("nan")
    need = lib.tk3d_chamfer_fwd_scratch_bytes(B, N, N, _lib.F32)
    assert 0 < need < (600 << 20) and need == lib.tk3d_chamfer_fwd_scratch_bytes(2 * B, N, N, _lib.F32)
    buf, res = torch.empty(need, dtype=torch.uint8, device=DEV), []
    for n in (0, need):
        d = [torch.empty(B, N, device=DEV) for _ in range(2)]
        i = [torch.empty(B, N, dtype=torch.int64, device=DEV) for _ in range(2)]
        sums = torch.empty(2, dtype=torch.float64, device=DEV)
        assert lib.tk3d_chamfer_fwd_ws(a.data_ptr(), b.data_ptr(), B, N, N, 0, d[0].data_ptr(), i[0].data_ptr(),
                                       d[1].data_ptr(), i[1].data_ptr(), sums.data_ptr(), buf.data_ptr(), n, _lib.F32,
                                       _stream()) == 0
        res.append(d + i + [sums])
    for x, y in zip(res[0][:4], res[1][:4]):
        assert _same(x, y)


@pytest.mark.parametrize("N,M,cf", [(1025, 4097, 0), (4096, 2048, 1), (1024, 20001, 1)])
@pytest.mark.parametrize("kind", ["uniform", "zeros", "nonfinite"])
def test_nothing_outside_the_scratch_and_the_outputs_is_written(kind, N, M, cf):
    from torkit3d_b200 import _lib

    lib = _lib.load()
    B, pad = 41, 4096
    a, b = _pair(kind, B, N, M, cf)

    def guarded(nbytes):
        t = torch.full((nbytes + 2 * pad,), 0x5A, dtype=torch.uint8, device=DEV)
        guards.append((t, nbytes))
        return t.data_ptr() + pad

    for k, ball in ((0, 0), (3, 0), (16, 0), (40, 0), (16, 1)):
        guards = []
        if k == 0:
            need = lib.tk3d_chamfer_fwd_scratch_bytes(B, N, M, _lib.F32)
            rc = lib.tk3d_chamfer_fwd_ws(a.data_ptr(), b.data_ptr(), B, N, M, cf, guarded(B * N * 4),
                                         guarded(B * N * 8), guarded(B * M * 4), guarded(B * M * 8), None,
                                         guarded(need), need, _lib.F32, _stream())
        elif ball:
            need = lib.tk3d_ball_query_scratch_bytes(B, N, M, k, _lib.F32)
            rc = lib.tk3d_ball_query_ws(a.data_ptr(), b.data_ptr(), B, N, M, 0.1, k, cf, guarded(B * N * k * 8),
                                        _lib.I64, guarded(need), need, _lib.F32, _stream())
        else:
            need = lib.tk3d_knn_scratch_bytes(B, N, M, k, _lib.F32)
            rc = lib.tk3d_knn_ws(a.data_ptr(), b.data_ptr(), B, N, M, k, cf, guarded(B * N * k * 4),
                                 guarded(B * N * k * 8), _lib.I64, guarded(need), need, _lib.F32, _stream())
        assert rc == 0 and need > 0
        for t, n in guards:
            assert bool((t[:pad] == 0x5A).all()) and bool((t[pad + n:] == 0x5A).all())

"""Gradients of the row gathers (csrc/scatter.cu) against float64 sums.

A gradient is a float32 sum of d terms in any order: its error is below d * 2^-24 times the sum of their magnitudes."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _index(kind, B, M, K, N):
    g = torch.Generator(device=DEV)
    g.manual_seed(M * K + N)
    i = torch.randint(0, N, (B, M, K), generator=g, device=DEV)
    if kind == "one":          # every entry the same target
        i[:] = N - 1
    elif kind == "padded":     # balls padded with their first hit, low indices first
        i[:, :, max(1, K // 3):] = (i[:, :, :1] // 7)
    elif kind == "hubs":       # a few targets with hundreds of entries, runs that cross pieces and slices
        i = torch.where(torch.rand(i.shape, generator=g, device=DEV) < 0.7, i % max(1, N // 50), i)
    elif kind == "bad":
        i[:, ::3, 0] = -1
        i[:, 1::5, K // 2] = N
    return i


def _scatter(g, index, N):
    """[B,C,M,K] -> sums and sums of magnitudes [B,C,N] in float64, entries per target [B,N]."""
    B, C = g.shape[:2]
    ok = (index >= 0) & (index < N)
    flat = torch.where(ok, index, N).reshape(B, 1, -1)
    g = g.double().reshape(B, C, -1)
    out = torch.zeros(B, C, N + 1, dtype=torch.float64, device=DEV)
    ex = flat.expand(-1, C, -1)
    count = torch.zeros(B, 1, N + 1, dtype=torch.float64, device=DEV).scatter_add_(2, flat, torch.ones_like(flat).double())
    return out.scatter_add(2, ex, g)[..., :N], out.scatter_add(2, ex, g.abs())[..., :N], count[..., :N]


def _close(got, ref, magnitude, count):
    bound = (count + 2) * 2.0 ** -24 * magnitude
    assert bool(((got.double() - ref).abs() <= bound).all())


SIZES = [  # B, C, N, M, K; sizes that are no multiples of 4 take this path from 1.2e7 elements on
    (1, 16, 1, 16, 16), (2, 20, 5, 36, 9), (3, 64, 31, 64, 16), (2, 131, 511, 771, 63), (3, 512, 64, 40, 16),
    (3, 129, 8192, 1024, 33), (2, 16, 100, 4096, 1), (1, 20, 700, 20, 1024), (1, 16, 4, 4, 1), (1, 38, 700, 350, 1000),
]


@pytest.mark.parametrize("kind", ["uniform", "one", "padded", "hubs", "bad"])
@pytest.mark.parametrize("B,C,N,M,K", SIZES)
def test_group(B, C, N, M, K, kind):
    from torkit3d_b200 import _lib

    lib = _lib.load()
    index = _index(kind, B, M, K, N)
    need = lib.tk3d_group_bwd_scratch_bytes(B, C, N, M, K, _lib.F32)
    assert need > 0
    raw = torch.randn(B * C * M * K + 3, device=DEV)
    for shift in (0, 1, 3):  # rows that start anywhere in a 16-byte line
        g = raw[shift:shift + B * C * M * K].view(B, C, M, K)
        out = torch.full((B, C, N), float("nan"), device=DEV)
        status = torch.zeros(1, dtype=torch.int32, device=DEV)
        scratch = torch.full((need,), 0xEE, dtype=torch.uint8, device=DEV)
        assert lib.tk3d_group_bwd(g.data_ptr(), index.data_ptr(), B, C, N, M, K, out.data_ptr(), status.data_ptr(),
                                  scratch.data_ptr(), need, _lib.F32, torch.cuda.current_stream().cuda_stream) == 0
        _close(out, *_scatter(g, index, N))
        assert int(status) == (1 if kind == "bad" else 0)


@pytest.mark.parametrize("kind", ["uniform", "padded", "bad"])
@pytest.mark.parametrize("cf", [True, False])
@pytest.mark.parametrize("B,C,N,M,K", [(2, 0, 40, 64, 8), (2, 6, 512, 128, 64), (4, 65, 333, 801, 61), (2, 3, 900, 700, 32)])
def test_set_abstraction(B, C, N, M, K, kind, cf):
    from torkit3d_b200 import _fused

    index = _index(kind, B, M, K, N)
    g = torch.randn(B, C + 3, M, K, device=DEV)
    ref, mag, count = _scatter(g, index, N)
    for wants in ((True, True, True), (True, False, False), (False, True, False)):
        feat, pts, cen = _fused.sa_group_backward(g, index.int(), C, N, channel_first=cf, need_feature=wants[0],
                                                  need_points=wants[1], need_centroids=wants[2])
        if wants[0] and C:
            _close(feat, ref[:, :C], mag[:, :C], count)
        if wants[1]:
            _close(pts if cf else pts.transpose(1, 2), ref[:, C:], mag[:, C:], count)
        if wants[2]:
            _close(cen if cf else cen.transpose(1, 2), -g[:, C:].double().sum(3), g[:, C:].double().abs().sum(3), K)


@pytest.mark.parametrize("kind", ["uniform", "hubs", "bad"])
@pytest.mark.parametrize("include_query", [True, False])
@pytest.mark.parametrize("B,C,N,M,K", [(2, 6, 300, 256, 8), (2, 64, 1024, 1024, 20), (6, 33, 777, 2051, 33), (1, 4, 50, 9000, 1), (1, 8, 70, 5, 200),
                                       (1, 200, 70, 5, 1000), (2, 100, 50, 63, 1001), (1, 2, 50, 90, 7)])
def test_edge(B, C, N, M, K, kind, include_query):
    from torkit3d_b200 import _fused

    index = _index(kind, B, M, K, N)
    g = torch.randn(B, 2 * C if include_query else C, M, K, device=DEV)
    ref, mag, count = _scatter(g[:, :C], index, N)
    q = -g[:, :C].double().sum(3) + (g[:, C:].double().sum(3) if include_query else 0)
    for need_query in (True, False):
        gq, gk = _fused.edge_feature_backward(g, index, C, N, include_query, need_query=need_query)
        _close(gk, ref, mag, count)
        if need_query:
            _close(gq, q, g.double().abs().sum(3).reshape(B, -1, C, M).sum(1), 2 * K)


@pytest.mark.parametrize("N", [65535 * 32 + 1, 65535 * 64 + 4])
def test_clouds_of_more_points_than_a_grid_has_rows(N):
    """The rows are written back point by point: no size of a grid may limit the points."""
    from torkit3d_b200 import _C, _fused

    M, K = -(-N // 64), 16
    index = _index("uniform", 1, M, K, N)
    index[0, 0] = N - 1
    g = torch.randn(1, 16, M, K, device=DEV)
    _close(_C.group_points_backward_cuda(g, index, N), *_scatter(g, index, N))
    index, g = index[:, :64].contiguous(), torch.randn(1, 8, 64, K, device=DEV)
    ref = _scatter(g[:, :4], index, N)
    _close(_fused.edge_feature_backward(g, index, 4, N)[1], *ref)
    _close(_fused.sa_group_backward(g[:, :7].contiguous(), index.int(), 4, N)[0], *ref)


@pytest.mark.parametrize("B,C,N,M,K", [(2, 37, 900, 4100, 41), (2, 64, 1024, 256, 16)])
def test_no_memory_for_the_rows(B, C, N, M, K, monkeypatch):
    """The rows are an option: where they cannot be allocated the direct kernels run."""
    from torkit3d_b200 import _C, _fused

    index = _index("padded", B, M, K, N)
    g = torch.randn(B, 2 * C, M, K, device=DEV)
    half, sa = g[:, :C].contiguous(), g[:, :C + 3].contiguous()
    ref = _scatter(half, index, N)
    empty, refused = torch.empty, []

    def none_for_scratch(*args, **kwargs):
        if kwargs.get("dtype") is torch.uint8:
            refused.append(args)
            raise torch.cuda.OutOfMemoryError("no memory")
        return empty(*args, **kwargs)

    monkeypatch.setattr(torch, "empty", none_for_scratch)
    got = (_C.group_points_backward_cuda(half, index, N), _fused.edge_feature_backward(g, index, C, N)[1],
           _fused.sa_group_backward(sa, index.int(), C, N)[0])
    monkeypatch.undo()
    assert len(refused) == 3
    for x in got:
        _close(x, *ref)


@pytest.mark.parametrize("kind", ["uniform", "padded", "bad"])
@pytest.mark.parametrize("B,C,N,M,K", [(4, 512, 300, 331, 16), (2, 64, 1000, 1303, 64), (2, 64, 1000, 1303, 60)])
def test_group_on_both_sides_of_the_folding_limit(B, C, N, M, K, kind):
    from torkit3d_b200 import _C

    index = _index(kind, B, M, K, N)
    g = torch.randn(B, C, M, K, device=DEV)
    _close(_C.group_points_backward_cuda(g, index, N), *_scatter(g, index, N))

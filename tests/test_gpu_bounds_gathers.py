"""The gathers of groups, their gradients, set abstraction and edge features through the range-checked build: no violation at
ragged sizes and the results of the regular build (sums that atomics make in any order: within their rounding)."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("B,C,N,M,K", [(2, 5, 257, 341, 7), (2, 64, 1024, 129, 16), (1, 131, 4099, 1101, 16), (3, 67, 300, 33, 41),
                                       (2, 4, 24577, 70, 16), (1, 12, 16400, 9001, 20), (2, 100, 50, 63, 129)])
def test_gathers(B, C, N, M, K):
    from torkit3d_b200 import _lib

    reg, chk = _lib.load(), _lib.load_bounds_checked()
    st = torch.cuda.current_stream().cuda_stream
    g = torch.Generator(device=DEV).manual_seed(N)
    index = torch.randint(0, N, (B, M, K), generator=g, device=DEV)
    index[:, :, K // 2:] = index[:, :, :1]
    i32 = index.int()
    f, q = torch.randn(B, C, N, generator=g, device=DEV), torch.randn(B, C, M, generator=g, device=DEV)
    p, c = torch.rand(B, 3, N, generator=g, device=DEV), torch.rand(B, 3, M, generator=g, device=DEV)
    grad = torch.randn(B, 2 * C + 3, M, K, generator=g, device=DEV)
    scratch = torch.empty(64 << 20, dtype=torch.uint8, device=DEV)
    before = chk.tk3d_bounds_violations()

    def new(*shape):
        return torch.full(shape, float("nan"), device=DEV)

    def both(fn, exact):
        for n in (scratch.numel(), 0):
            a, b = fn(reg, scratch.data_ptr() if n else None, n), fn(chk, scratch.data_ptr() if n else None, n)
            for x, y in zip(a, b):
                assert torch.equal(x, y) if exact else torch.allclose(x, y, rtol=1e-4, atol=1e-3)

    def group(lib, s, n):
        out = new(B, C, M, K)
        assert lib.tk3d_group_fwd(f.data_ptr(), index.data_ptr(), B, C, N, M, K, out.data_ptr(), None, s, n, _lib.F32, st) == 0
        return (out,)

    def group_bwd(lib, s, n):
        out = new(B, C, N)
        assert lib.tk3d_group_bwd(grad.data_ptr(), index.data_ptr(), B, C, N, M, K, out.data_ptr(), None, s, n, _lib.F32,
                                  st) == 0
        return (out,)

    def edge(lib, s, n):
        out = new(B, 2 * C, M, K)
        assert lib.tk3d_edge_feature_fwd(q.data_ptr(), f.data_ptr(), index.data_ptr(), B, C, M, N, K, 1, out.data_ptr(), None,
                                         s, n, _lib.F32, st) == 0
        return (out,)

    def edge_bwd(lib, s, n):
        gq, gk = new(B, C, M), new(B, C, N)
        assert lib.tk3d_edge_feature_bwd(grad.data_ptr(), index.data_ptr(), B, C, M, N, K, 1, gq.data_ptr(), gk.data_ptr(),
                                         None, s, n, _lib.F32, st) == 0
        return gq, gk

    def sa(lib, s, n):
        out, i = new(B, C + 3, M, K), torch.empty(B, M, K, dtype=torch.int32, device=DEV)
        if K <= 128 and n:
            assert lib.tk3d_sa_group_fwd(p.data_ptr(), c.data_ptr(), f.data_ptr(), B, C, N, M, 0.2, K, 1, 1, out.data_ptr(),
                                         i.data_ptr(), None, s, n, _lib.F32, st) == 0
        return (out, i) if K <= 128 and n else ()

    def sa_bwd(lib, s, n):
        out = new(B, C, N), new(B, 3, N), new(B, 3, M)
        if K <= 128:
            assert lib.tk3d_sa_group_bwd(grad.data_ptr(), i32.data_ptr(), B, C, N, M, K, 1, 1, *(o.data_ptr() for o in out),
                                         None, s, n, _lib.F32, st) == 0
        return out if K <= 128 else ()

    for fn, exact in ((group, True), (edge, True), (sa, True), (group_bwd, False), (edge_bwd, False), (sa_bwd, False)):
        both(fn, exact)
    assert chk.tk3d_bounds_violations() == before

"""Gathers by channel rows (csrc/chanrow.cuh) at row and output alignments of every kind: results are exact copies
(set abstraction: one rounded subtraction), compared with advanced indexing."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _gather(f, index):
    """[B,C,N], [B,M,K] -> [B,C,M,K]; an index outside [0,N) reads 0."""
    B, C, N = f.shape
    f = torch.cat([f, torch.zeros(B, C, 1, dtype=f.dtype, device=DEV)], 2)
    flat = torch.where((index >= 0) & (index < N), index, N).long().reshape(B, 1, -1).expand(-1, C, -1)
    return f.gather(2, flat).reshape(B, C, *index.shape[1:])


@pytest.mark.parametrize("dt", [torch.float32, torch.float64])
@pytest.mark.parametrize("B,C,N,M,K", [(2, 3, 256, 64, 16), (1, 5, 257, 341, 3), (3, 17, 1023, 129, 33), (2, 9, 4099, 1025, 8),
                                       (1, 2, 12288, 9000, 1), (1, 3, 24575, 700, 6), (33, 20, 2050, 300, 30)])
def test_group(B, C, N, M, K, dt):
    from torkit3d_b200 import _lib

    lib = _lib.load()
    code = _lib.F32 if dt == torch.float32 else _lib.F64
    index = torch.randint(-1, N + 1, (B, M, K), device=DEV)
    index[0, 0, 0] = -1
    raw = torch.randn(B * C * N + 3, dtype=dt, device=DEV)
    out_raw = torch.empty(B * C * M * K + 3, dtype=dt, device=DEV)
    for shift in (0, 1, 3):  # rows and outputs that start anywhere in a 16-byte line
        f = raw[shift:shift + B * C * N].view(B, C, N)
        out_raw.fill_(float("nan"))
        out = out_raw[shift:shift + B * C * M * K].view(B, C, M, K)
        for ix, t in ((index, _lib.I64), (index.int(), _lib.I32)):
            status = torch.zeros(1, dtype=torch.int32, device=DEV)
            assert lib.tk3d_group_fwd_layout(f.data_ptr(), ix.data_ptr(), t, B, C, N, M, K, out.data_ptr(), status.data_ptr(),
                                             None, 0, code, torch.cuda.current_stream().cuda_stream) == 0
            assert torch.equal(out, _gather(f, index)) and int(status) == 1
            assert bool(out_raw[:shift].isnan().all()) and bool(out_raw[shift + B * C * M * K:].isnan().all())


@pytest.mark.parametrize("cf", [True, False])
@pytest.mark.parametrize("use_xyz", [True, False])
@pytest.mark.parametrize("want_index", [True, False])
@pytest.mark.parametrize("B,C,N,M,K", [(2, 6, 256, 64, 16), (1, 0, 300, 70, 16), (3, 131, 1023, 129, 33), (2, 7, 24575, 63, 17),
                                       (9, 5, 16384, 1500, 8), (2, 4, 24577, 64, 16), (2, 4, 100, 64, 16)])
def test_set_abstraction(B, C, N, M, K, cf, use_xyz, want_index):
    """Equal to the ball query and the centred gather one by one, on both sides of the limits of the two-step path."""
    from torkit3d_b200 import _C, _fused

    if C == 0 and not use_xyz:
        return
    g = torch.Generator(device=DEV)
    g.manual_seed(N)
    p = torch.rand(B, 3, N, generator=g, device=DEV)
    q = torch.cat([p[:, :, :M - 2], torch.full((B, 3, 2), 9.0, device=DEV)], 2).contiguous()  # two centres without a hit
    f = torch.randn(B, C, N, generator=g, device=DEV) if C else None
    radius = 1.2 * (K / N) ** (1 / 3) / 2
    a, c = (p, q) if cf else (p.transpose(1, 2).contiguous(), q.transpose(1, 2).contiguous())
    out, index = _fused.sa_group_forward(a, c, f, radius, K, use_xyz=use_xyz, channel_first=cf, want_index=want_index)
    ref = _C.ball_query_cuda(c, a, radius, K, channel_first=cf)
    parts = ([_gather(f, ref)] if C else []) + ([_gather(p, ref) - q.unsqueeze(-1)] if use_xyz else [])
    assert torch.equal(out, torch.cat(parts, 1))
    if want_index:
        assert torch.equal(index.long(), ref)


@pytest.mark.parametrize("dt", [torch.float32, torch.float64])
@pytest.mark.parametrize("B,C,N,M,K", [(2, 40, 1023, 1300, 33), (1, 131, 4099, 1101, 16), (1, 12, 12287, 11201, 17),
                                       (3, 1, 301, 44667, 15), (64, 3, 257, 345, 31), (1, 64, 255, 1024, 31)])
def test_rows_in_pieces(B, C, N, M, K, dt):
    """Outputs large enough for rows that are no whole 16-byte lines; nothing beside the output is written."""
    from torkit3d_b200 import _lib

    lib = _lib.load()
    index = torch.randint(-1, N + 1, (B, M, K), device=DEV)
    index[0, 0, 0] = N
    n = B * C * M * K
    raw = torch.randn(B * C * N + 3, dtype=dt, device=DEV)
    out_raw = torch.empty(n + 64, dtype=dt, device=DEV)
    for shift in (0, 1, 3):
        f = raw[shift:shift + B * C * N].view(B, C, N)
        out_raw.fill_(7.5)
        out = out_raw[32 + shift:32 + shift + n].view(B, C, M, K)
        status = torch.zeros(1, dtype=torch.int32, device=DEV)
        assert lib.tk3d_group_fwd(f.data_ptr(), index.data_ptr(), B, C, N, M, K, out.data_ptr(), status.data_ptr(), None, 0,
                                  _lib.F32 if dt == torch.float32 else _lib.F64,
                                  torch.cuda.current_stream().cuda_stream) == 0
        assert torch.equal(out, _gather(f, index)) and int(status) == 1
        assert bool((out_raw[:32 + shift] == 7.5).all()) and bool((out_raw[32 + shift + n:] == 7.5).all())

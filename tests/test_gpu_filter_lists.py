"""What the tensor cores' filter of feature-space neighbours finds (csrc/feature_filter.cu), read from its scratch: the
results alone cannot tell, since every query it leaves is redone by the kernel they are compared with."""
import ctypes

import pytest
import torch

from test_gpu_feature_filter import _features, _run

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _filter(q, r, k):
    """-> distances, indices, lists [B,N1,2,64], their lengths [B,N1,2], counts [B,N1]."""
    from torkit3d_b200 import _lib

    lib = _lib.load()
    B, C, N1, N2 = q.size(0), q.size(1), q.size(2), r.size(2)
    same = q.data_ptr() == r.data_ptr()
    need = lib.tk3d_feature_knn_scratch_bytes(max(B, 40), max(C, 16), max(N1, 640), max(N2, 512), k, _lib.F32)
    assert need > 0
    scratch = torch.full((need,), 0xEE, dtype=torch.uint8, device=DEV)
    d = torch.empty(B, N1, k, device=DEV)
    i = torch.empty(B, N1, k, dtype=torch.int64, device=DEV)
    assert lib.tk3d_feature_knn_ws(q.data_ptr(), r.data_ptr(), B, C, N1, N2, k, 1, d.data_ptr(), i.data_ptr(),
                                   scratch.data_ptr(), need, _lib.F32, torch.cuda.current_stream().cuda_stream) == 0
    off = (ctypes.c_size_t * 3)()
    assert lib.tk3d_diag_feature_filter(B, C, N1, N2, k, 1 if same else 0, off) == 0

    def view(at, n, dt, size):
        return scratch[at:at + n * size].view(dt)

    lists = view(off[0], B * N1 * 128, torch.int16, 2).view(B, N1, 2, 64).int() & 0xFFFF
    return d, i, lists, view(off[1], B * N1 * 2, torch.int32, 4).view(B, N1, 2), \
        view(off[2], B * N1, torch.int32, 4).view(B, N1)


def _check(q, r, k):
    """Every query with a list has its k nearest in it; -> share of the queries that have none."""
    from torkit3d_b200 import _lib

    d, i, lists, length, counts = _filter(q, r, k)
    ref = _run(_lib.load(), _lib, q, r, k, True, False)
    have = counts >= 0
    assert torch.equal(counts[have], length.sum(2)[have].int())
    listed = torch.where(torch.arange(64, device=DEV) < length.unsqueeze(3), lists, -1).flatten(2)[have]
    wanted = ref[1][have]
    for part in range(0, wanted.size(0), 4096):
        w, l = wanted[part:part + 4096], listed[part:part + 4096]
        assert bool((w.unsqueeze(2) == l.unsqueeze(1)).any(2).all())
    assert torch.equal(d[have], ref[0][have]) and torch.equal(i[have], ref[1][have])
    return 1 - have.float().mean().item()


@pytest.mark.parametrize("kind", ["normal", "relu", "offset", "scales", "sorted"])
@pytest.mark.parametrize("C,N,k", [(64, 1024, 20), (16, 2000, 16), (128, 700, 20), (33, 1030, 8)])
def test_no_query_is_left(C, N, k, kind):
    x = _features(kind, 2, C, N, 3)
    assert _check(x, x, k) == 0
    assert _check(_features(kind, 2, C, 300, 4), x, k) < (0.5 if kind in ("scales", "sorted") else 1e-9)


@pytest.mark.parametrize("C", [1, 2, 3, 5])
@pytest.mark.parametrize("kind", ["normal", "relu", "offset", "scales", "outlier", "sorted"])
def test_few_channels(C, kind):
    """Where the halves' error is nearest to its bound."""
    for N, k in ((1024, 20), (4096, 5)):
        x = _features(kind, 2, C, N, 5)
        _check(x, x, k)
        _check(_features(kind, 2, C, 300, 6), x, k)


@pytest.mark.parametrize("kind", ["outlier", "lattice", "periodic"])
def test_few_queries_are_left(kind):
    x = _features(kind, 2, 64, 1024, 3)
    assert _check(x, x, 20) <= 0.1


@pytest.mark.parametrize("kind", ["same", "tiny", "overflow", "nan"])
def test_clouds_that_are_left(kind):
    x = _features(kind, 2, 64, 1024, 3)
    counts = _filter(x, x, 20)[4]
    assert bool((counts[0] < 0).all()) and (kind == "nan" or bool((counts[1] < 0).all()))
    assert kind != "nan" or bool((counts[1] >= 0).all())


def test_groups_are_left_as_a_whole():
    """One query far from the keys: its group has no other query with a result of the filter, the other groups all."""
    x = _features("normal", 1, 64, 1024, 3)
    q = x.clone()
    q[0, :, 77] = 1e6
    counts = _filter(q, x, 20)[4][0]
    assert bool((counts[64:96] < 0).all()) and bool((counts[:64] >= 0).all()) and bool((counts[96:] >= 0).all())

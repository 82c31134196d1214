"""Feature-space neighbours at the edges of the kernel's tiles, bit for bit against the oracle.

Key tiles hold 256 points, slices 16 channels, a block 32 queries, lists 32, 64 or 128 entries; the
channel-first copies are 16 bytes wide where sizes and alignment allow and 4 bytes otherwise.  Candidates
are merged 32 at a time: ties, more than a buffer of equal distances, +inf and NaN distances included.
"""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _run(q, r, k, cf):
    from torkit3d_b200 import _C

    d, i = _C.feature_knn_cuda(q, r, k, channel_first=cf)
    return d.cpu().numpy(), i.cpu().numpy()


@pytest.mark.parametrize("cf", [False, True])
@pytest.mark.parametrize("C,n1,n2,k", [(1, 1, 1, 1), (15, 31, 255, 32), (16, 32, 256, 32), (17, 33, 257, 33),
                                       (33, 64, 512, 64), (16, 36, 516, 65), (3, 5, 1000, 128)])
@pytest.mark.parametrize("values", ["normal", "few", "same"])
def test_tile_edges(oracle, cf, C, n1, n2, k, values):
    g = np.random.default_rng(C + n1 + n2)
    shape = (lambda n: (2, C, n)) if cf else (lambda n: (2, n, C))
    if values == "normal":
        q, r = (g.standard_normal(shape(n)).astype(np.float32) for n in (n1, n2))
    elif values == "few":  # distances take a handful of values: ties go to the lower index
        q, r = (g.integers(0, 2, shape(n)).astype(np.float32) for n in (n1, n2))
    else:
        q, r = (np.full(shape(n), 0.5, np.float32) for n in (n1, n2))
    d, i = _run(torch.from_numpy(q).to(DEV), torch.from_numpy(r).to(DEV), k, cf)
    e, j = oracle.feature_knn(q, r, k, channel_first=cf)
    assert np.array_equal(d, e) and np.array_equal(i, j)


def test_unaligned_tensors_take_the_narrow_copies():
    g = torch.Generator().manual_seed(3)
    buf = torch.randn(1 + 2 * 20 * 300, generator=g).to(DEV)
    x = buf[1:].view(2, 20, 300)  # contiguous, four bytes off a 16-byte boundary
    d, i = _run(x, x, 20, True)
    e, j = _run(x.clone(), x.clone(), 20, True)
    assert np.array_equal(d, e) and np.array_equal(i, j)


def test_infinite_distances_rank_last_and_nan_never():
    x = torch.zeros(1, 40, 4)
    x[0, :, 0] = torch.arange(40)
    x[0, 10, 0], x[0, 11, 0] = float("inf"), float("nan")
    d, i = _run(x[:, :1].contiguous().to(DEV), x.to(DEV), 40, False)
    order = [j for j in range(40) if j not in (10, 11)]
    assert i[0, 0].tolist() == order + [10, -1]
    assert d[0, 0, :38].tolist() == [float(j * j) for j in order] and np.isinf(d[0, 0, 38:]).all()


def test_point_major_rows_are_staged_without_bank_conflicts():
    """Staging point-major tensors costs strided reads, not bank conflicts (with them 1.85 times the channel-first call)."""
    from torkit3d_b200 import _C

    g = torch.Generator(device=DEV).manual_seed(0)
    a = torch.randn(4, 128, 4096, generator=g, device=DEV)
    p = a.transpose(1, 2).contiguous()

    def us(fn):
        best = float("inf")
        for _ in range(6):
            e0, e1 = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            e0.record()
            fn()
            e1.record()
            torch.cuda.synchronize()
            best = min(best, e0.elapsed_time(e1) * 1e3)
        return best

    assert us(lambda: _C.feature_knn_cuda(p, p, 40, channel_first=False)) < 1.6 * us(lambda: _C.feature_knn_cuda(a, a, 40))

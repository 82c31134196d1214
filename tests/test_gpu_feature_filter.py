"""Feature-space neighbours with candidates from the tensor cores (csrc/feature_filter.cu) equal those of the kernel that
evaluates every pair, bit for bit: the matrix product only decides which pairs are evaluated."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _run(lib, L, q, r, k, cf, filtered):
    B, N1, N2 = q.size(0), q.size(2 if cf else 1), r.size(2 if cf else 1)
    C = q.size(1 if cf else 2)
    # the size for a large batch holds the small ones that the rule leaves to the other kernel
    need = lib.tk3d_feature_knn_scratch_bytes(max(B, 40), C, max(N1, 640), max(N2, 512), k, L.F32) if filtered else 0
    assert not filtered or need > 0
    scratch = torch.full((max(need, 1),), 0xEE, dtype=torch.uint8, device=DEV)
    d = torch.full((B, N1, k), float("nan"), device=DEV)
    i = torch.full((B, N1, k), -7, dtype=torch.int64, device=DEV)
    assert lib.tk3d_feature_knn_ws(q.data_ptr(), r.data_ptr(), B, C, N1, N2, k, 1 if cf else 0, d.data_ptr(), i.data_ptr(),
                                   scratch.data_ptr() if need else None, need, L.F32,
                                   torch.cuda.current_stream().cuda_stream) == 0
    return d, i


def _features(kind, B, C, N, seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    x = torch.randn(B, C, N, generator=g, device=DEV)
    if kind == "relu":
        x = torch.relu(x) + 0.1 * x
    elif kind == "offset":      # far from the origin
        x = x + 100
    elif kind == "scales":      # channels and points of very different size
        x = x * torch.logspace(-3, 2, C, device=DEV).view(1, -1, 1) * torch.logspace(-1, 1, N, device=DEV)
    elif kind == "lattice":     # ties
        x = torch.randint(0, 2, x.shape, generator=g, device=DEV).float()
    elif kind == "same":        # every point the same
        x = x[:, :, :1].expand(-1, -1, N).contiguous()
    elif kind == "tiny":
        x = x * 1e-21
    elif kind == "huge":
        x = x * 1e18
    elif kind == "overflow":    # norms beyond the largest number
        x = x * 1e20
    elif kind == "nan":
        x[0, C // 2, N // 3] = float("nan")
    elif kind == "inf":
        x[0, 0, 5] = float("inf")
        x[-1, C - 1, N - 1] = -float("inf")
    elif kind == "outlier":
        x[:, :, 7] *= 1e4
    elif kind == "periodic":    # neighbours are 32 apart
        x = x[:, :, :32].repeat(1, 1, -(-N // 32))[:, :, :N] * 10 + 0.1 * x
    elif kind == "sorted":      # neighbours follow one another in memory
        x = torch.cumsum(0.1 * x, 2)
    return x


def _equal(a, b):
    assert torch.equal(a[1], b[1])
    assert torch.equal(a[0].nan_to_num(nan=-1.0), b[0].nan_to_num(nan=-1.0))


@pytest.mark.parametrize("cf", [True, False])
@pytest.mark.parametrize("B,C,N1,N2,k", [(1, 16, 128, 256, 8), (2, 64, 300, 1024, 20), (1, 1, 5, 257, 1), (3, 33, 129, 511, 48),
                                         (1, 128, 640, 2048, 33), (2, 17, 1000, 300, 32), (1, 3, 200, 65536, 7)])
def test_equals_every_pair(B, C, N1, N2, k, cf):
    from torkit3d_b200 import _lib

    q, r = _features("normal", B, C, N1, 1), _features("normal", B, C, N2, 2)
    if not cf:
        q, r = q.transpose(1, 2).contiguous(), r.transpose(1, 2).contiguous()
    lib = _lib.load()
    _equal(_run(lib, _lib, q, r, k, cf, True), _run(lib, _lib, q, r, k, cf, False))
    if N1 == 300:  # queries that are the keys
        _equal(_run(lib, _lib, r, r, k, cf, True), _run(lib, _lib, r, r, k, cf, False))


@pytest.mark.parametrize("kind", ["relu", "offset", "scales", "lattice", "same", "tiny", "huge", "overflow", "nan", "inf",
                                  "outlier", "sorted", "periodic"])
def test_inputs_of_every_kind(kind):
    from torkit3d_b200 import _lib

    lib = _lib.load()
    for C, N, k in ((64, 1024, 20), (40, 700, 40)):
        x = _features(kind, 2, C, N, 3)
        _equal(_run(lib, _lib, x, x, k, True, True), _run(lib, _lib, x, x, k, True, False))


def test_no_access_out_of_range():
    from torkit3d_b200 import _lib

    lib = _lib.load_bounds_checked()
    before = lib.tk3d_bounds_violations()
    for kind in ("normal", "lattice", "nan", "overflow", "inf"):
        x = _features(kind, 2, 40, 700, 3)
        _equal(_run(lib, _lib, x, x, 40, True, True), _run(lib, _lib, x, x, 40, True, False))
    assert lib.tk3d_bounds_violations() == before

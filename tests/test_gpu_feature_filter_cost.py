"""What the tensor cores' filter of feature-space neighbours costs on inputs it does not serve, and that few far points do not
keep it from serving the others: against the same entry point without scratch, which evaluates all pairs."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
B, C, N, K = 32, 64, 1024, 20


def _features(kind):
    g = torch.Generator(device=DEV).manual_seed(3)
    x = torch.randn(B, C, N, generator=g, device=DEV)
    if kind == "equal":
        x = x[:, :, :1].expand(-1, -1, N).contiguous()
    elif kind == "tiny":
        x *= 1e-21
    elif kind == "nan":
        x[:, C // 2, N // 3] = float("nan")
    elif kind == "clusters":  # eight, far apart against their size
        pick = torch.randint(0, 8, (N,), generator=g, device=DEV)
        x = 0.01 * x + torch.randn(B, C, 8, generator=g, device=DEV)[:, :, pick]
    elif kind == "far":       # one point 100 times as far out as the others
        x[:, :, 7] *= 100
    elif kind == "very far":  # and one of the points that the centre is made of
        x[:, :, N // 8] *= 1e4
    elif kind == "scales":
        x *= torch.logspace(-3, 2, C, device=DEV).view(1, -1, 1) * torch.logspace(-1, 1, N, device=DEV)
    return x


def _times(kind):
    from torkit3d_b200 import _lib

    lib = _lib.load()
    x = _features(kind)
    need = lib.tk3d_feature_knn_scratch_bytes(B, C, N, N, K, _lib.F32)
    assert need > 0
    scratch = torch.empty(need, dtype=torch.uint8, device=DEV)
    d, i = torch.empty(B, N, K, device=DEV), torch.empty(B, N, K, dtype=torch.int64, device=DEV)
    times, out = [], []
    for n in (0, need):
        def run():
            assert lib.tk3d_feature_knn_ws(x.data_ptr(), x.data_ptr(), B, C, N, N, K, 1, d.data_ptr(), i.data_ptr(),
                                           scratch.data_ptr(), n, _lib.F32, torch.cuda.current_stream().cuda_stream) == 0
        best = float("inf")
        for _ in range(8):
            a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            a.record()
            for _ in range(4):
                run()
            b.record()
            torch.cuda.synchronize()
            best = min(best, a.elapsed_time(b) * 1e3 / 4)
        times.append(best)
        out.append((d.nan_to_num(nan=-1.0), i.clone()))
    assert torch.equal(out[0][0], out[1][0]) and torch.equal(out[0][1], out[1][1])
    return times


@pytest.mark.parametrize("kind", ["equal", "tiny", "nan", "clusters"])
def test_looking_in_vain(kind):
    plain, filtered = _times(kind)
    assert filtered < 1.15 * plain + 15


@pytest.mark.parametrize("kind", ["far", "very far", "scales"])
def test_few_far_points_are_no_reason_to_give_up(kind):
    plain, filtered = _times(kind)
    assert filtered < 0.85 * plain

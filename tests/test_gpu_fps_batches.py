"""Cluster FPS, where one exchange yields several samples: the sequence is the oracle's, index by index.

Sizes cover every cluster shape (one, two and four candidates per lane; coordinates in registers and in
shared memory); the inputs what ends a batch early: exact ties within and between warps, duplicates whose
distances run out, a sample next to the following candidate, more samples than one batch holds.
"""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _cloud(kind, B, N):
    g = np.random.default_rng(N)
    if kind == "random":
        return g.random((B, N, 3), dtype=np.float32)
    if kind == "lattice":
        return g.integers(0, 7, (B, N, 3)).astype(np.float32) * np.float32(0.25)
    if kind == "few":  # 40 distinct points, then only zero distances
        return g.random((B, 40, 3), dtype=np.float32)[:, g.integers(0, 40, N)]
    if kind == "far":  # a handful of far points among near ones: long batches, then none
        p = g.random((B, N, 3), dtype=np.float32) * np.float32(0.01)
        p[:, ::997] += g.standard_normal((B, len(range(0, N, 997)), 3)).astype(np.float32) * 10
        return p
    p = g.random((B, N, 3), dtype=np.float32)  # sorted along x: neighbours share a warp
    return np.take_along_axis(p, np.argsort(p[..., :1], axis=1, kind="stable"), axis=1)


@pytest.mark.parametrize("kind", ["random", "lattice", "few", "far", "sorted"])
@pytest.mark.parametrize("B,N,S", [(2, 4097, 200), (1, 8192, 300), (2, 8193, 100), (1, 16385, 150), (1, 40000, 90),
                                   (1, 65537, 90), (1, 131073, 60)])
def test_sequence(oracle, kind, B, N, S):
    from torkit3d_b200.ops import sample_farthest_points

    p = np.ascontiguousarray(_cloud(kind, B, N))
    got = sample_farthest_points(torch.from_numpy(p).to(DEV), S).cpu().numpy()
    np.testing.assert_array_equal(got, oracle.fps(p, S))


@pytest.mark.parametrize("kind", ["random", "lattice", "few", "far", "sorted"])
@pytest.mark.parametrize("B,N,S", [(2, 4097, 200), (2, 8193, 100), (1, 16385, 150), (1, 40000, 90), (1, 65537, 90)])
def test_sequence_of_batches_whatever_the_number_of_samples(oracle, kind, B, N, S):
    """The diagnostic entry takes several samples per exchange also where a regular call takes one (few samples)."""
    from torkit3d_b200 import _lib

    p = np.ascontiguousarray(_cloud(kind, B, N))
    pts = torch.from_numpy(p).to(DEV)
    idx = torch.empty(B, S, dtype=torch.int64, device=DEV)
    assert _lib.load().tk3d_diag_fps_wait_limit(pts.data_ptr(), B, N, S, idx.data_ptr(), 1000, -1,
                                                torch.cuda.current_stream().cuda_stream) == 0
    np.testing.assert_array_equal(idx.cpu().numpy(), oracle.fps(p, S))


@pytest.mark.parametrize("B,N", [(32, 8192), (16, 20000), (2, 131072)])
def test_few_samples_do_not_pay_for_bounds(B, N):
    """64 samples: a regular call is faster than the one that takes several samples per exchange (0.72 to 0.84 of it)."""
    from torkit3d_b200 import _lib
    from torkit3d_b200.ops import sample_farthest_points

    pts = torch.rand(B, N, 3, generator=torch.Generator(device=DEV).manual_seed(N), device=DEV)
    idx = torch.empty(B, 64, dtype=torch.int64, device=DEV)
    st = torch.cuda.current_stream().cuda_stream

    def several():
        assert _lib.load().tk3d_diag_fps_wait_limit(pts.data_ptr(), B, N, 64, idx.data_ptr(), 1000, -1, st) == 0

    def us(fn):
        best = float("inf")
        for _ in range(10):
            e0, e1 = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            torch.cuda.synchronize()
            torch.cuda._sleep(200000)  # the host is ahead: the launch is not part of the time
            e0.record()
            fn()
            e1.record()
            torch.cuda.synchronize()
            best = min(best, e0.elapsed_time(e1) * 1e3)
        return best

    assert us(lambda: sample_farthest_points(pts, 64)) < 0.95 * us(several)

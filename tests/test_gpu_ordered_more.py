"""Searches over spatially ordered clouds, continued: a cloud searched in itself, clouds that are away from one another,
collapsed, or so far apart that distances overflow, batches of which only some clouds are ordered, sums of cut batches,
memory that is short, a device that refuses the cluster launch."""
import os
import subprocess
import sys
import textwrap

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _stream():
    return torch.cuda.current_stream().cuda_stream


def _same(x, y):
    return torch.equal(x.view(torch.int32) if x.dtype == torch.float32 else x,
                       y.view(torch.int32) if y.dtype == torch.float32 else y)


def _knn(a, b, k, cf, scratch):
    from torkit3d_b200 import _lib

    B, N, M = a.shape[0], a.shape[2 if cf else 1], b.shape[2 if cf else 1]
    d, i = torch.empty(B, N, k, device=DEV), torch.empty(B, N, k, dtype=torch.int64, device=DEV)
    assert _lib.load().tk3d_knn_ws(a.data_ptr(), b.data_ptr(), B, N, M, k, cf, d.data_ptr(), i.data_ptr(), _lib.I64,
                                   scratch.data_ptr() if scratch is not None else None,
                                   scratch.numel() if scratch is not None else 0, _lib.F32, _stream()) == 0
    return d, i


def _chamfer(a, b, scratch):
    from torkit3d_b200 import _lib

    B, N, M = a.shape[0], a.shape[1], b.shape[1]
    out = [torch.empty(B, n, dtype=t, device=DEV) for n in (N, M) for t in (torch.float32, torch.int64)]
    sums = torch.empty(2, dtype=torch.float64, device=DEV)
    assert _lib.load().tk3d_chamfer_fwd_ws(a.data_ptr(), b.data_ptr(), B, N, M, 0, *(o.data_ptr() for o in out),
                                           sums.data_ptr(), scratch.data_ptr() if scratch is not None else None,
                                           scratch.numel() if scratch is not None else 0, _lib.F32, _stream()) == 0
    return out + [sums]


@pytest.mark.parametrize("kind", ["random", "lattice", "zeros", "outlier", "nonfinite"])
@pytest.mark.parametrize("k", [1, 3, 4, 5, 16, 32, 64])
@pytest.mark.parametrize("B,N,cf", [(2, 1024, 0), (3, 1025, 1), (1, 8200, 0)])
def test_a_cloud_searched_in_itself(kind, k, B, N, cf):
    g = torch.Generator().manual_seed(N)
    p = torch.randn(B, N, 3, generator=g)
    if kind == "lattice":
        p = torch.randint(0, 9, (B, N, 3), generator=g).float() * 0.1
    elif kind == "zeros":
        p[torch.rand(B, N, generator=g) < 0.3] = 0
    elif kind == "outlier":
        p[:, N // 2] = 1e6
    elif kind == "nonfinite":
        p[B - 1, 7, 1] = float("nan")
    p = (p.transpose(1, 2).contiguous() if cf else p).to(DEV)
    scratch = torch.full((32 << 20,), 0xA5, dtype=torch.uint8, device=DEV)
    for x, y in zip(_knn(p, p, k, cf, None), _knn(p, p, k, cf, scratch)):
        assert _same(x, y)


@pytest.mark.parametrize("kind", ["away", "collapsed", "inside", "overflow", "halves"])
@pytest.mark.parametrize("B,N,M", [(2, 1030, 4099), (1, 4096, 1024)])
def test_clouds_that_lie_badly_to_each_other(kind, B, N, M):
    g = torch.Generator().manual_seed(M)
    a, b = torch.randn(B, N, 3, generator=g), torch.randn(B, M, 3, generator=g)
    if kind == "away":
        a += 100
    elif kind == "collapsed":
        a[:] = 0.25
    elif kind == "inside":
        a *= 1e-3
        b /= b.norm(dim=2, keepdim=True)
    elif kind == "overflow":  # finite coordinates, infinite distances: no nearest neighbour in the chamfer distance
        a -= 3e19
        b += 3e19
    else:  # half of the queries like the keys, half away: some lists are short, some long
        a[:, ::2] += 50
    a, b = a.to(DEV), b.to(DEV)
    scratch = torch.full((32 << 20,), 0xA5, dtype=torch.uint8, device=DEV)
    for x, y in zip(_chamfer(a, b, None)[:4], _chamfer(a, b, scratch)[:4]):
        assert _same(x, y)
    for k in (1, 3, 5, 16, 40, 64):
        for x, y in zip(_knn(a, b, k, 0, None), _knn(a, b, k, 0, scratch)):
            assert _same(x, y)


@pytest.mark.parametrize("bad", [(0,), (1,), (2,), (0, 2)])
def test_weights_of_a_batch_of_which_some_clouds_are_swept(bad):
    from torkit3d_b200 import _fused, ops

    B, C, N, M = 3, 4, 11000, 4100
    g = torch.Generator(device=DEV).manual_seed(5)
    a, b = torch.randn(B, 3, N, generator=g, device=DEV), torch.randn(B, 3, M, generator=g, device=DEV)
    for i in bad:
        b[i, 1, 77] = float("inf")
    f = torch.randn(B, C, M, generator=g, device=DEV)
    _, index, weight = _fused.three_nn_interp_forward(a, b, f)
    for q0 in range(0, N, 2000):  # too few pairs to be ordered
        d, i = ops.knn_points(a[:, :, q0:q0 + 2000].contiguous(), b, 3, transpose=True)
        assert torch.equal(index[:, q0:q0 + 2000].long(), i)
        assert _same(weight[:, q0:q0 + 2000].contiguous(), ops.three_nn_weight(d))


def test_sums_of_a_batch_that_is_cut():
    from torkit3d_b200 import _lib

    B, N = 9001, 1024  # built in two parts
    g = torch.Generator(device=DEV).manual_seed(1)
    a, b = (torch.randn(B, N, 3, generator=g, device=DEV) for _ in range(2))
    a[4000, 3], a[B - 1, 5] = 1e4, 1e4  # one swept cloud in each part
    need = _lib.load().tk3d_chamfer_fwd_scratch_bytes(B, N, N, _lib.F32)
    x, y = _chamfer(a, b, None), _chamfer(a, b, torch.empty(need, dtype=torch.uint8, device=DEV))
    for p, q in zip(x[:4], y[:4]):
        assert _same(p, q)
    torch.testing.assert_close(x[4], y[4], rtol=1e-12, atol=0)


@pytest.mark.parametrize("op", ["chamfer", "knn", "ball", "interp", "sa", "step"])
def test_calls_sweep_where_the_memory_for_the_order_is_missing(op):
    """The order takes scratch that a sweep does not: a call that just fits without it still runs."""
    from torkit3d_b200 import _fused, _lib, dist, ops

    B, N = 64, 16384
    g = torch.Generator(device=DEV).manual_seed(2)
    a, b = (torch.rand(B, N, 3, generator=g, device=DEV) for _ in range(2))
    acf, bcf = (t.transpose(1, 2).contiguous() for t in (a, b))
    f = torch.randn(B, 2, N, generator=g, device=DEV)
    run = {
        "chamfer": lambda: ops.nn_distance(a, b),
        "knn": lambda: ops.knn_points(a, b, 3),
        "ball": lambda: [ops.ball_query(a, b, 0.02, 4, transpose=False)],
        "interp": lambda: _fused.three_nn_interp_forward(acf, bcf, f),
        "sa": lambda: _fused.sa_group_forward(bcf, acf, f, 0.02, 4),
        "step": lambda: dist.chamfer_step(a, b),
    }[op]
    margin = 28 << 20
    assert _lib.scratch_bytes("tk3d_chamfer_fwd", B, N, N, _lib.F32) > margin + (12 << 20)
    want = list(run())
    results = sum(t.numel() * t.element_size() for t in want)
    if op == "step":  # distances and indices are temporaries
        results += 2 * B * N * 12
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    total = torch.cuda.get_device_properties(0).total_memory
    torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + results + margin) / total)
    try:
        got = list(run())
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
    for x, y in zip(want, got):
        if op == "step":
            torch.testing.assert_close(x, y, rtol=1e-5, atol=1e-9)  # float32 sums in any order
        else:
            assert _same(x, y)


def test_a_device_that_refuses_the_cluster_launch_is_swept(tmp_path):
    """The cluster launch of the sort is made to fail on the host, by a stand-in for the runtime call."""
    src = tmp_path / "refuse.c"
    src.write_text(textwrap.dedent("""
        #define _GNU_SOURCE
        #include <dlfcn.h>
        #include <cuda_runtime.h>
        typedef cudaError_t (*launch_t)(const cudaLaunchConfig_t *, const void *, void **);
        cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *c, const void *f, void **a) {
          for (unsigned i = 0; i < c->numAttrs; ++i)
            if (c->attrs[i].id == cudaLaunchAttributeClusterDimension) return cudaErrorInvalidClusterSize;
          return ((launch_t)dlsym(RTLD_NEXT, "cudaLaunchKernelExC"))(c, f, a);
        }
    """))
    so = tmp_path / "refuse.so"
    subprocess.run(["gcc", "-shared", "-fPIC", "-I/usr/local/cuda/include", "-o", str(so), str(src), "-ldl"], check=True)
    code = textwrap.dedent("""
        import sys
        sys.path.insert(0, %r)
        import torch
        from torkit3d_b200 import _fused, _lib, ops
        g = torch.Generator(device="cuda").manual_seed(3)
        a, b = (torch.rand(2, 9000, 3, generator=g, device="cuda") for _ in range(2))
        assert _lib.scratch_bytes("tk3d_chamfer_fwd", 2, 9000, 9000, _lib.F32) > 0
        out = list(ops.nn_distance(a, b))
        for k in (3, 16):
            out += ops.knn_points(a, b, k)
        out.append(ops.ball_query(a, b, 0.05, 16, transpose=False))
        acf, bcf = (t.transpose(1, 2).contiguous() for t in (a, b))
        f = torch.randn(2, 4, 9000, generator=g, device="cuda")
        out += _fused.three_nn_interp_forward(acf, bcf, f)
        out += _fused.sa_group_forward(bcf, acf, f, 0.05, 8)
        torch.save([t.cpu() for t in out], sys.argv[1])
    """ % ROOT)
    res = []
    for name, env in (("plain", {}), ("refused", {"LD_PRELOAD": str(so)})):
        path = tmp_path / name
        p = subprocess.run([sys.executable, "-c", code, str(path)], env={**os.environ, **env}, capture_output=True, text=True,
                           timeout=300)
        assert p.returncode == 0, p.stderr[-2000:]
        res.append(torch.load(path))
    for x, y in zip(*res):
        assert _same(x, y)

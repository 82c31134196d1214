"""Searches over spatially ordered clouds, continued: memory that is short, a device that refuses the cluster launch."""
import os
import subprocess
import sys
import textwrap

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _same(x, y):
    return torch.equal(x.view(torch.int32) if x.dtype == torch.float32 else x,
                       y.view(torch.int32) if y.dtype == torch.float32 else y)


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

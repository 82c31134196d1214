"""Searches over spatially ordered clouds, continued: a device that refuses the cluster launch."""
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

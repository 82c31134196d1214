"""Which problems the library asks scratch for, i.e. orders the clouds of (host logic, no GPU needed)."""


def test_few_queries_among_many_keys_are_swept():
    from torkit3d_b200 import _lib

    lib = _lib.load()
    for B, N, M, k in ((1, 1000, 100000, 3), (8, 512, 16384, 3), (2, 4096, 32768, 3), (16, 1024, 4096, 1),
                       (1, 64, 400000, 16), (16, 128, 65536, 32)):
        assert lib.tk3d_knn_scratch_bytes(B, N, M, k, _lib.F32) == 0
    for B, N, M in ((4, 1024, 16384), (4, 1024, 65536), (1, 2048, 65536), (1, 65536, 2048)):
        assert lib.tk3d_chamfer_fwd_scratch_bytes(B, N, M, _lib.F32) == 0
    for B, N, M in ((16, 512, 16384), (4, 2048, 65536), (1, 300, 400000)):
        assert lib.tk3d_ball_query_scratch_bytes(B, N, M, 32, _lib.F32) == 0
    assert lib.tk3d_knn_scratch_bytes(16, 4096, 4096, 3, _lib.F32) > 0
    assert lib.tk3d_knn_scratch_bytes(1, 2048, 16384, 16, _lib.F32) > 0
    assert lib.tk3d_chamfer_fwd_scratch_bytes(24, 2500, 4099, _lib.F32) > 0
    assert lib.tk3d_ball_query_scratch_bytes(32, 1024, 8192, 32, _lib.F32) > 0

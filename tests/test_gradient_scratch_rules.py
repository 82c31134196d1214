"""Which gradients of the row gathers the library asks scratch for (host logic, no GPU needed)."""


def test_very_large_clouds():
    """Clouds beyond the transposition's grid take the rows where there are channels and entries enough for them."""
    from torkit3d_b200 import _lib

    lib, F32 = _lib.load(), _lib.F32
    edge, most = 65535 * 32, (1 << 30) - 1
    for C, N, M, K in ((16, edge + 1, 131072, 16), (32, 2 * edge + 4, 131072, 16), (16, most, 1 << 25, 16)):
        want = 4 * C * N
        assert lib.tk3d_group_bwd_scratch_bytes(1, C, N, M, K, F32) == want
        assert lib.tk3d_edge_feature_bwd_scratch_bytes(1, C, M, N, K, F32) == want
        assert lib.tk3d_sa_group_bwd_scratch_bytes(1, C, N, M, K, F32) == want
    for C, N, M, K in ((12, edge + 4, 131072, 16), (16, edge + 1, 1024, 16), (64, most, 1024, 16)):
        assert lib.tk3d_group_bwd_scratch_bytes(1, C, N, M, K, F32) == 0
        assert lib.tk3d_edge_feature_bwd_scratch_bytes(1, C, M, N, K, F32) == 0
        assert lib.tk3d_sa_group_bwd_scratch_bytes(1, C, N, M, K, F32) == 0
    # up to the grid's limit as for any cloud
    assert lib.tk3d_edge_feature_bwd_scratch_bytes(1, 4, 1024, edge, 16, F32) == 4 * 4 * edge
    assert lib.tk3d_sa_group_bwd_scratch_bytes(1, 4, edge, 1024, 16, F32) == 4 * 4 * edge


def test_set_abstraction_with_short_odd_lists():
    """Few elements whose lists are no multiple of four run the direct kernel: the rows cost more launches than they save."""
    from torkit3d_b200 import _lib

    lib, F32 = _lib.load(), _lib.F32
    for B, C, N, M, K in ((1, 100, 328, 104, 2), (5, 44, 7613, 772, 1), (12, 4, 9071, 5324, 5)):
        assert lib.tk3d_sa_group_bwd_scratch_bytes(B, C, N, M, K, F32) == 0
    for B, C, N, M, K in ((5, 188, 2943, 1390, 2), (1, 100, 328, 104, 4), (4, 8, 8675, 2870, 14), (2, 64, 512, 128, 16)):
        assert lib.tk3d_sa_group_bwd_scratch_bytes(B, C, N, M, K, F32) == 4 * B * C * N

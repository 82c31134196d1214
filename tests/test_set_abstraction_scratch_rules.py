"""How much scratch the set-abstraction front end asks for (host logic, no GPU needed)."""


def test_the_neighbours_have_a_place_where_no_index_is_wanted():
    """Neighbours first, then the gather: without an index tensor their lists go to scratch, in the place of the features' rows."""
    from torkit3d_b200 import _lib

    lib, F32 = _lib.load(), _lib.F32
    for B, C, N, M, K in ((2, 16, 4096, 2048, 64), (1, 3, 1024, 512, 32), (4, 8, 1024, 256, 64), (1, 0, 2048, 1024, 32)):
        assert M * K > C * N
        assert lib.tk3d_sa_group_scratch_bytes(B, C, N, M, K, F32) == 4 * B * M * K
    for B, C, N, M, K in ((2, 64, 4096, 512, 32), (1, 128, 1024, 256, 16)):  # the rows are larger
        assert lib.tk3d_sa_group_scratch_bytes(B, C, N, M, K, F32) == 4 * B * C * N
    for B, C, N, M, K in ((2, 6, 200, 100, 64), (1, 3, 25000, 2000, 64), (1, 6, 300, 30, 32)):  # the fused kernel
        assert lib.tk3d_sa_group_scratch_bytes(B, C, N, M, K, F32) == 4 * B * C * N
    # clouds that are ordered: rows, search and lists
    assert lib.tk3d_sa_group_scratch_bytes(32, 64, 8192, 1024, 32, F32) > 4 * 32 * (64 * 8192 + 1024 * 32)

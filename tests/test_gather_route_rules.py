"""Which gathers of groups the library asks scratch for, i.e. makes from transposed rows (host logic, no GPU needed)."""


def test_rows_by_points_and_by_channels():
    from torkit3d_b200 import _lib

    lib, F32 = _lib.load(), _lib.F32
    for C, N, M, K in ((64, 8192, 4096, 32), (64, 24000, 6000, 64), (64, 4879, 4879, 4), (131, 20411, 20411, 16),
                       (64, 20411, 1276, 16)):
        assert lib.tk3d_group_fwd_scratch_bytes(8, C, N, M, K, F32) == 0
    # odd rows, many entries per point, sizes for 16-byte accesses
    for C, N, M, K in ((64, 4879, 2440, 32), (64, 20411, 20412, 4), (16, 8191, 4096, 16)):
        assert lib.tk3d_group_fwd_scratch_bytes(8, C, N, M, K, F32) == 4 * 8 * C * N
    # odd rows and too little output for rows in pieces
    assert lib.tk3d_group_fwd_scratch_bytes(1, 64, 1185, 296, 16, F32) == 4 * 64 * 1185

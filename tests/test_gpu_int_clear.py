"""The integer product clears its result before it adds to it: results that held something else, sizes around those of the
clearing kernel's blocks and of a launch (32 rows), and calls that follow one another with and without programmatic launches."""
import numpy as np
import pytest
import torch

import decode_matmul_b200 as dmm
from oracle import dmm_oracle as o

pytestmark = pytest.mark.gpu


# Both ways of clearing: a memset below 32 tiles of 256 rows x 32 k per SM, a kernel from there on (9472 x 4096: 32 exactly, 37888 x 1056:
# 33), with fewer and with more 16-byte pieces than the kernel has threads, and with two launches of the product.
@pytest.mark.parametrize("M,N,K", [(1, 16, 96), (5, 208, 96), (65, 9488, 96), (8, 16, 32768), (1, 9472, 4096), (1, 37888, 1056), (33, 37888, 1056)])
@pytest.mark.parametrize("pdl", [False, True])
def test_result_that_held_something(M, N, K, pdl):
    rng = np.random.default_rng(M + N)
    cb = np.ascontiguousarray(o.build_codebook_abs())
    codes = rng.integers(-32768, 32768, size=(N, K // 8)).astype(np.int16)
    w, cbd = torch.from_numpy(o.tile_pack(codes)).cuda(), torch.from_numpy(cb).cuda()
    out = torch.full((M, N), 12345, dtype=torch.int32, device="cuda")
    for i in range(3):  # each call overwrites what the one before left
        x = rng.integers(-128, 128, size=(M, K)).astype(np.int8)
        y = dmm.decode_matmul_i8(torch.from_numpy(x).cuda(), w, cbd, out, pdl=pdl)
        assert y.data_ptr() == out.data_ptr()
        assert np.array_equal(y.cpu().numpy(), o.decode_matmul_int(x, codes, cb))
    assert dmm.status() == 0

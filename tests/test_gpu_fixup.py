"""Tiles whose reduction is split over CTAs: one tile over all of them, few units, ragged ends, and the counters that the shared
fix-up leaves behind.  Needs a B200."""
import numpy as np
import pytest
import torch

import decode_matmul_b200 as dmm
from oracle import dmm_oracle as o

pytestmark = pytest.mark.gpu


# (rows, N, K): one tile over every CTA, and one row block of it; tiles that share CTAs; both sides of the line for sharing (at 64
# rows 4096 and 28672 output rows); rows that leave the last 16 columns ragged; the builds that never share
@pytest.mark.parametrize("M,N,K", [(64, 16, 32768), (64, 256, 28672), (33, 4096, 2080), (50, 5120, 1056), (64, 28672, 544),
                                   (17, 272, 8192), (100, 4096, 2080), (128, 256, 28672), (333, 2816, 4096)])
def test_split_tiles(M, N, K):
    rng = np.random.default_rng(M + N + K)
    codes = rng.integers(-32768, 32768, size=(N, K // 8)).astype(np.int16)
    cb16 = o.synthetic_codebook(42)
    w = torch.from_numpy(o.decode_weights_f16(codes, cb16)).cuda().double()
    tiled, cb = torch.from_numpy(o.tile_pack(codes)).cuda(), torch.from_numpy(cb16).cuda()
    small = torch.randn((64, 32), device="cuda").half()
    for seed in range(3):
        x = torch.randn((M, K), generator=torch.Generator().manual_seed(seed)).half().cuda()
        want = x.double() @ w.T
        y = dmm.decode_matmul_fp16(x, tiled, cb)
        # the error of sums cut after 88 MMAs, see test_gpu_wide.py
        assert float((y.double() - want).norm() / want.norm()) <= 1e-6
        assert torch.equal(y, dmm.decode_matmul_fp16(x, tiled, cb)), "the summation order must not depend on who adds up"
        # another shape in between, with its own split, on the same workspace
        dmm.decode_matmul_fp16(small, tiled[:16, :4].contiguous(), cb)
    assert dmm.status() == 0

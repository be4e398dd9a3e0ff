"""Tiles whose reduction is split over CTAs: one tile over many of them, few units, ragged ends, and the counters that the shared
fix-up leaves behind.  Needs a B200."""
import numpy as np
import pytest
import torch

import decode_matmul_b200 as dmm
from oracle import dmm_oracle as o

pytestmark = pytest.mark.gpu


# (rows, N, K): one tile over 16 CTAs, and one row block of it; tiles that share CTAs; tiles of few units, which stay whole; rows
# that leave the last 16 columns ragged; the builds that never share
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


# The shared fix-up has a mapping of rows of its own for the fast layout, and adds to what the output holds: one tile over 16 CTAs, and
# tiles that share CTAs (33 to 64 rows, more than 150 KiB of parts).
@pytest.mark.parametrize("M,N,K", [(64, 256, 28672), (33, 4096, 2080), (64, 4096, 2080), (50, 5120, 5120)])
@pytest.mark.parametrize("fast", [False, True])
@pytest.mark.parametrize("accumulate", [False, True])
def test_shared_tiles(M, N, K, fast, accumulate):
    rng = np.random.default_rng(M + N + K)
    codes = rng.integers(-32768, 32768, size=(N, K // 8)).astype(np.int16)
    cb16 = o.synthetic_codebook(42)
    packed, cb = torch.from_numpy(o.fast_pack(codes) if fast else o.tile_pack(codes)).cuda(), torch.from_numpy(cb16).cuda()
    w = torch.from_numpy(o.decode_weights_f16(codes, cb16)).cuda().double()
    x = torch.randn((M, K), generator=torch.Generator().manual_seed(K)).half().cuda()
    base = torch.randn((M, N), device="cuda")
    want = x.double() @ w.T + (base.double() if accumulate else 0.0)
    layout = dmm.LAYOUT_FAST if fast else dmm.LAYOUT_TILE
    got = [dmm.decode_matmul_fp16(x, packed, cb, 1.0, base.clone(), layout=layout, accumulate=accumulate) for _ in range(2)]
    # as above, and one more rounding where the product is added to something
    assert float((got[0].double() - want).norm() / want.norm()) <= 1.1e-6
    assert torch.equal(got[0], got[1])
    assert dmm.status() == 0


# The small-batch kernels' own fix-up, eight parts at a time: 5 to 6 parts per super-tile, 9 to 10, 18 to 19, 37 and all 148, loads beyond the
# last part included (the workspace holds NaN where nothing was written); rows that the loaders split and, at 8 rows 9600 x 8192, planes.
@pytest.mark.parametrize("N,K", [(8192, 3072), (4096, 4096), (2048, 2048), (1024, 4096), (16, 32768), (9600, 8192)])
@pytest.mark.parametrize("M", [1, 2, 3, 5, 8])
def test_split_super_tiles(M, N, K):
    gen = torch.Generator(device="cuda").manual_seed(M + N + K)
    codes = torch.randint(-32768, 32768, (N, K // 8), dtype=torch.int16, device="cuda", generator=gen)
    cb = torch.from_numpy(o.synthetic_codebook(42)).cuda()
    x = torch.randn((M, K), device="cuda", generator=gen)
    want = x.half().double() @ dmm.decode_weights(codes, cb).double().T
    ws = torch.full((dmm.workspace_bytes(M, N, K),), 255, dtype=torch.uint8, device="cuda")
    ws[:1024] = 0  # the counters
    got = []
    for _ in range(2):
        y = torch.full((M, N), float("nan"), device="cuda")
        dmm.decode_matmul_fused(x, codes, cb, 1.0, y, workspace=ws)
        # exact products, sums off by the truncation of the tensor core: 7e-7 to 9e-7 at any length
        assert float((y.double() - want).norm() / want.norm()) <= 2e-6
        got.append(y)
    assert torch.equal(got[0], got[1])
    assert dmm.status() == 0

"""Calls of different sizes that share one workspace: what one leaves there must not reach the next.  Needs a B200."""
import pytest
import torch

import decode_matmul_b200 as dmm
from decode_matmul_b200 import _lib
from oracle import dmm_oracle as o

pytestmark = pytest.mark.gpu


def _product(M, N, K, path):
    gen = torch.Generator(device="cuda").manual_seed(N + K)
    codes = torch.randint(-32768, 32768, (N, K // 8), dtype=torch.int16, device="cuda", generator=gen)
    cb = torch.from_numpy(o.synthetic_codebook(42)).cuda()
    x = torch.randn((M, K), device="cuda", generator=gen).to(torch.float16)
    y = torch.full((M, N), float("nan"), device="cuda")  # what is not written shows
    dmm.decode_matmul_fp16(x, codes, cb, 1.0, y, path=path)
    w = dmm.decode_weights(codes, cb)
    want = torch.cat([x.double() @ part.double().T for part in w.split(65536)], dim=1)
    return float((y.double() - want).norm() / want.norm())


# Few rows and a long reduction leave partial sums from the start of the workspace on; many rows after them need one
# counter per split tile, which has to be zero.  (The widest layout of the counters is that of the last kernel.)
@pytest.mark.parametrize("path,M,large", [(_lib.PATH_AUTO, 1, (1 << 20, 128)), (_lib.PATH_AUTO, 8, (1 << 20, 128)),
                                          (_lib.PATH_AUTO, 24, (57344, 1024)), (_lib.PATH_TCGEN05, 1, (1 << 20, 128)),
                                          (_lib.PATH_GEMV, 1, (57344, 2048)), (_lib.PATH_GEMV, 16, (57344, 2048))])
def test_many_rows_after_few(path, M, large):
    for small in (16, 256, 4096):
        assert _product(M, small, 32768, path) <= 1e-4
        # K terms are at most 2048: 1.5e-5 as in the tests of the single kernels; NaN where a tile was never written
        assert _product(M, *large, path) <= 1.5e-5
    assert dmm.status() == 0

"""The activations of the fp8-plane kernels, split by the product's own loaders or by the kernel in front of it: runs of k-tiles that
cross the end of a row (also several times), ragged epochs, every input kind, both sides of the line.  Needs a B200."""
import numpy as np
import pytest
import torch

import decode_matmul_b200 as dmm
from decode_matmul_b200 import _lib
from oracle import dmm_oracle as o

pytestmark = pytest.mark.gpu

# Activations and weights are exact in the planes; what is left are the fp32 sums.  An addition is off by at most 2^-23 of the running
# sum (the tensor core truncates): 128 of them at the very worst by 128 * 2^-23 = 1.5e-5, and the errors of more grow slower than
# that.  (With few terms a single large one decides: 1.4e-6 at K = 32.)  A piece in the wrong place is off by 1, a
# lost fourth plane by some 1e-4.
REL = 1.5e-5


def _inputs(kind, M, K, seed):
    g = torch.Generator().manual_seed(seed)
    if kind == "half":
        x = torch.randn((M, K), generator=g).half()
        return x, x.double(), dict(x_kind=_lib.X_F16)
    if kind == "float":
        x = torch.randn((M, K), generator=g)
        return x, x.half().double(), dict(x_kind=_lib.X_F32)
    x = torch.randn((M, 2 * K), generator=g)
    return x, (torch.nn.functional.silu(x[:, :K]) * x[:, K:]).half().double(), dict(x_kind=_lib.X_F32_SILU_MUL, k=K, x_gap=K)


# K = 32 and 96: a run of k-tiles crosses the end of the row at every (third) tile; 38400 and 37904 rows are 150 and 149 super-tiles,
# one or two per CTA.  4096 x 1056: some three tiles per CTA, an epoch is never full.  9600 x 8192: 65 tiles per SM, where the
# loaders split up to 6 rows and the kernel in front 7 and 8.
@pytest.mark.parametrize("N,K", [(38400, 32), (37904, 96), (4096, 1056), (9600, 8192)])
@pytest.mark.parametrize("M", [1, 2, 3, 4, 6, 7, 8])
@pytest.mark.parametrize("kind", ["half", "float", "silu"])
def test_split(kind, M, N, K):
    rng = np.random.default_rng(N + K)
    codes = rng.integers(-32768, 32768, size=(N, K // 8)).astype(np.int16)
    cb16 = o.synthetic_codebook(42)
    tiled, cb = torch.from_numpy(o.tile_pack(codes)).cuda(), torch.from_numpy(cb16).cuda()
    w = dmm.decode_weights(tiled, cb).double()  # (bit-exact against the oracle: test_gpu_parity.py)
    x, half, kw = _inputs(kind, M, K, M)
    want = half.cuda() @ w.T
    out = torch.zeros((M, N), device="cuda")
    dmm.decode_matmul_fused(x.cuda(), tiled, cb, 1.0, out, accumulate=True, atomic=True, **kw)
    # silu in the kernel uses the fast exponential: its rounding to half can differ by an ulp here and there
    assert float((out.double() - want).norm() / want.norm()) <= (1e-4 if kind == "silu" else REL)
    assert dmm.status() == 0


# The slots form of the tensor-parallel step in a group of one: rows 4 to 8, where producer and consumer both split in their loaders
# (no launch besides the four products of a block and the last sum), and a down projection of 67 tiles per SM, beyond the line of 8 rows.
@pytest.mark.parametrize("batch,hidden,ffn,extra", [(4, 2048, 5632, 0), (5, 1024, 2816, 0), (6, 2048, 5632, 0), (8, 2048, 5632, 0), (8, 5632, 14336, 1)])
def test_slots_form(batch, hidden, ffn, extra):
    from decode_matmul_b200.linear import LinearStack

    cfg = dict(hidden=hidden, kv_heads=4, head_dim=128, ffn=ffn, layers=2)
    cb = dmm.synthetic_codebook(42)
    plain = LinearStack(cfg, cb, "cuda", logical_seed=12, scale=2.0 ** -9)
    slots = LinearStack(cfg, cb, "cuda", logical_seed=12, scale=2.0 ** -9, tp_mode="slots")
    torch.manual_seed(batch)
    for step in range(3):  # the epoch counter and the slot parities carry over
        h0 = torch.randn(batch, hidden, device="cuda")
        want = plain.step(h0.clone(), fused=True)
        before = dmm.launch_count()
        got = slots.step(h0.clone(), fused=True)
        if step > 0 and torch.cuda.get_device_properties(0).multi_processor_count == 148:
            assert dmm.launch_count() - before == (4 + extra) * cfg["layers"] + 1
        assert dmm.status() == 0
        # an activation whose sum comes out one bit lower can round to another half: as for the form at 1 and 3 rows
        assert torch.allclose(got, want, rtol=2e-3, atol=2e-3), f"step {step}: {float((got - want).abs().max())}"


# The integer kernel's loaders copy one piece per thread where an epoch has no more than 64 of them, else four: few rows and few tiles,
# runs of k-tiles that cross the end of a row, epochs of exactly 64 pieces (2 * tiles * rows) and of a few more.
@pytest.mark.parametrize("N,K", [(37904, 96), (65536, 32), (4096, 1056), (16, 32768), (9600, 2080)])
@pytest.mark.parametrize("M", [1, 2, 4, 8, 13, 16, 17, 32])
def test_integer_loaders(M, N, K):
    gen = torch.Generator(device="cuda").manual_seed(M + N + K)
    codes = torch.randint(-32768, 32768, (N, K // 8), dtype=torch.int16, device="cuda", generator=gen)
    cb = dmm.build_codebook_abs("cuda")
    x = torch.randint(-128, 128, (M, K), dtype=torch.int8, device="cuda", generator=gen)
    base = torch.randint(-1000, 1000, (M, N), dtype=torch.int32, device="cuda", generator=gen)
    want = (x.double() @ dmm.decode_weights(codes, cb).double().T).to(torch.int32)  # (whole numbers below 2^53: exact)
    assert torch.equal(dmm.decode_matmul_i8(x, codes, cb), want)
    assert torch.equal(dmm.decode_matmul_i8(x, codes, cb, base.clone(), accumulate=True), base + want)
    assert dmm.status() == 0

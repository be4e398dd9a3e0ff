"""decode_matmul_sequence on the GPU: the same as its products one by one, and what an error leaves behind."""
import pytest
import torch

import decode_matmul_b200 as dmm
from decode_matmul_b200 import _lib, ops
from decode_matmul_b200.linear import DecodeLinear
from oracle import dmm_oracle as o

pytestmark = pytest.mark.gpu


def _layers(shapes):
    gen = torch.Generator(device="cuda").manual_seed(3)
    cb = torch.from_numpy(o.synthetic_codebook(42)).cuda()
    return [DecodeLinear(torch.randint(-32768, 32768, (n, k // 8), dtype=torch.int16, device="cuda", generator=gen), cb, 2.0 ** -7)
            for n, k in shapes]


@pytest.mark.parametrize("M", [1, 5, 16, 24])
def test_same_as_the_products_one_by_one(M):
    first, second = _layers([(544, 1056), (1056, 544)])
    x = torch.randn((M, 1056), device="cuda")
    a, y = torch.zeros((M, 544), device="cuda"), torch.zeros((M, 1056), device="cuda")
    ops.decode_matmul_sequence([ops.fused_op(x, first, a), ops.fused_op(a, second, y)], M, x.device)
    a1 = torch.zeros_like(a)
    dmm.decode_matmul_fused(x, first.codes, first.codebook, first.scale, a1, accumulate=True, atomic=True)
    y1 = torch.zeros_like(y)
    dmm.decode_matmul_fused(a, second.codes, second.codebook, second.scale, y1, accumulate=True, atomic=True)
    # the same kernels over the same inputs: only the order of the atomic adds differs, a few roundings of 2^-24
    for got, want in ((a, a1), (y, y1)):
        assert float((got - want).norm() / want.norm()) <= 4 * 2.0 ** -24
    assert dmm.status() == 0


# Products that would go different ways by themselves share one: at 6 rows the loaders split although 138 tiles per SM lie beyond
# their line, at 8 rows planes_kernel runs in front of a product of 13 tiles per SM too.
@pytest.mark.parametrize("M,shapes,launches", [(6, [(544, 1056), (20480, 8192)], 2), (8, [(4096, 4096), (28672, 8192)], 4)])
def test_one_choice_for_all_products(M, shapes, launches):
    layers = _layers(shapes)
    xs = [torch.randn((M, k), device="cuda") for _, k in shapes]
    ys = [torch.zeros((M, n), device="cuda") for n, _ in shapes]
    before = dmm.launch_count()
    ops.decode_matmul_sequence([ops.fused_op(x, lin, y) for x, lin, y in zip(xs, layers, ys)], M, xs[0].device)
    if torch.cuda.get_device_properties(0).multi_processor_count == 148:
        assert dmm.launch_count() - before == launches
    for x, lin, y in zip(xs, layers, ys):
        w = dmm.decode_weights(lin.codes, lin.codebook)
        want = torch.cat([x.half().double() @ part.double().T for part in w.split(8192)], dim=1) * lin.scale
        # exact products, sums off by the truncation of the tensor core: 7e-7 to 9e-7 at any length
        assert float((y.double() - want).norm() / want.norm()) <= 2e-6
    assert dmm.status() == 0


def test_an_error_in_the_middle():
    """The ops before the refused one have been launched, the ones behind it have not, and no hint is left for the next
    call."""
    good, last = _layers([(544, 1056), (1056, 544)])
    M = 2
    x = torch.randn((M, 1056), device="cuda")
    a, y = torch.zeros((M, 544), device="cuda"), torch.full((M, 1056), 3.0, device="cuda")
    bad = _layers([(48, 544)])[0]
    bad.codes = bad.codes[:24].contiguous()  # 24 rows: not a multiple of 16
    block = [ops.fused_op(x, good, a), ops.fused_op(a, bad, torch.zeros((M, 24), device="cuda")), ops.fused_op(a, last, y)]
    with pytest.raises(RuntimeError, match="decode_matmul_sequence"):
        ops.decode_matmul_sequence(block, M, x.device)
    want = torch.zeros_like(a)
    dmm.decode_matmul_fused(x, good.codes, good.codebook, good.scale, want, accumulate=True, atomic=True)
    assert float((a - want).norm() / want.norm()) <= 4 * 2.0 ** -24
    assert bool((y == 3.0).all())
    # an op in the middle whose codes are missing altogether, through the C entry
    arr = (_lib.FusedOp * 2)(block[0][0], block[2][0])
    arr[1].codes = None
    a.zero_()
    rc = _lib.lib().dmm_f16_sequence(arr, 2, M, _lib.SIGN_SLOW, _lib.FLAG_ACCUMULATE | _lib.FLAG_ATOMIC, None, 0, 0, None, 0,
                                     torch.cuda.current_stream().cuda_stream)
    assert rc == -1
    assert float((a - want).norm() / want.norm()) <= 4 * 2.0 ** -24
    assert dmm.status() == 0

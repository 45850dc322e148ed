"""The stand-alone product of a few rows on weights that are fetched into shared memory as a whole, in slices of K: the bits of the
shape-generic kernel at the edges of its shares, slices and rows, and either side of the lines of its rule."""
import pytest
import torch

import quant_ops_b200 as q
from helpers import N, abi_int4_matmul, launched_kernels, lib, stream_ptr

pytestmark = pytest.mark.gpu
DEV = "cuda:0"

# rows; K of one slice less than four, four whole ones, a last slice of one chunk of 128 and of a few; one channel per CTA, the most
# channels, a last CTA with fewer; rows, channels or K past each line
SHAPES = [(9, 4096, 4096, True), (32, 4096, 148, True), (16, 14336, 4096, True), (17, 8320, 1000, True), (32, 6144, 4736, True), (4, 11008, 4095, True),
          (5, 14336, 200, True), (31, 2048, 2368, True), (12, 4224, 333, True), (9, 16384, 2000, True), (8, 4096, 4096, False), (16, 4096, 4737, False),
          (3, 11008, 4096, False), (31, 2048, 2369, False), (32, 1920, 1000, False), (9, 4096, 147, False), (16, 98304, 1000, False)]


@pytest.mark.parametrize("t,k,n,resident", SHAPES)
def test_same_bits_as_the_generic_kernel(t, k, n, resident):
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("the lines are given for 148 SMs")
    g = torch.Generator(device=DEV).manual_seed(t + k + n)
    words = lambda *s: torch.randint(-2 ** 31, 2 ** 31, s, dtype=torch.int64, device=DEV, generator=g).to(torch.int32)
    a, w = words(t, k // 8), words(n, k // 8)
    sa, sb = torch.rand(t, device=DEV, generator=g) + 0.01, torch.rand(n, device=DEV, generator=g) * 1e-3
    for out_dtype in ("fp16", "bf16"):
        ref, ref_acc = abi_int4_matmul(a, w.t(), sa, sb, out_dtype, True, policy=1)
        for _ in range(3):
            got, acc = abi_int4_matmul(a, w.t(), sa, sb, out_dtype, True)
            assert torch.equal(acc, ref_acc) and torch.equal(got.view(torch.int16), ref.view(torch.int16))
    wide = torch.zeros(n, k // 8 + 4, dtype=torch.int32, device=DEV)  # weights with a larger row stride
    wide[:, :k // 8] = w
    assert torch.equal(abi_int4_matmul(a, wide[:, :k // 8].t(), sa, sb, "bf16").view(torch.int16), ref.view(torch.int16))
    assert lib.qo_device_status(stream_ptr()) == N.QO_OK
    assert ("int4_gemm_resident_kernel" in launched_kernels(lambda: q.int4_matmul(a, w.t(), sa, sb))[0]) == resident

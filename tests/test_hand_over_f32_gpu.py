"""float32 quantizer and dequantizer launch beside the end of the kernel ahead: queues of them on the same buffers, with inputs that change,
see what that kernel wrote and overwrite nothing that it still reads."""
import pytest
import torch

from helpers import N, QD, lib, make_inputs, ptr, stream_ptr

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
CALLS = 120


@pytest.mark.parametrize("pack", [True, False])
@pytest.mark.parametrize("tokens,feat", [(3, 4096), (400, 4096), (70, 14336)])
def test_quantize_then_dequantize(tokens, feat, pack):
    inputs = [tuple(v.to(DEV) for v in make_inputs(tokens, feat, "fp32", seed=i)) for i in range(3)]
    m, n = inputs[0][1].shape[0], inputs[0][2].shape[0]
    x, codes = torch.zeros(tokens, feat, device=DEV), torch.zeros(tokens, feat // 8 if pack else feat, dtype=torch.int32 if pack else torch.int8, device=DEV)
    scales, back = torch.zeros(tokens, device=DEV), torch.zeros(tokens, feat, device=DEV)

    def quantize(i):
        _, left, right = inputs[i % 3]
        N.check(lib.qo_flatquant_quantize(ptr(x), feat, ptr(left), ptr(right), ptr(codes), ptr(scales), tokens, m, n, 0.9, QD["fp32"], int(pack),
                                          QD["fp32"], stream_ptr()))

    def dequantize(out):
        N.check(lib.qo_dequantize_int4(ptr(codes), ptr(scales), ptr(out), tokens, feat, int(pack), QD["fp32"], stream_ptr()))

    want = []
    for i in range(3):
        x.copy_(inputs[i][0])
        quantize(i)
        torch.cuda.synchronize()
        dequantize(back)
        torch.cuda.synchronize()
        want.append(back.clone())
    outs = [torch.zeros_like(back) for _ in range(CALLS)]
    torch.cuda.synchronize()
    for i in range(CALLS):
        x.copy_(inputs[i % 3][0])
        quantize(i)
        dequantize(outs[i])
    torch.cuda.synchronize()
    wrong = [i for i in range(CALLS) if not torch.equal(outs[i], want[i % 3])]
    assert not wrong, wrong

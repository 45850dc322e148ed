"""GPU parity of the quantizer for right transforms of 144 .. 256 (flatquant_sm100_n256.cu), at the edges of its tiles: against the
oracle, and against the SIMT kernel on tokens with infinities, NaNs and zeros."""
import ctypes as C

import pytest
import torch

from helpers import N, abi_quantize, lib, make_inputs, ptr, QD, stream_ptr, t2f, TD
from oracle import w4a4_oracle as O
from test_quantize_gpu import check

pytestmark = pytest.mark.gpu
DEV = "cuda:0"

# (M, N): both halves of the rows or one, 32-column blocks whole or half, the second tile's lanes from 16 to 128;
# tokens: one, a few, more than one round of every SM
WIDE = [(128, 224, "bf16", 1, True), (128, 224, "fp16", 150, False), (128, 256, "bf16", 301, True), (16, 144, "bf16", 40, True),
        (16, 256, "fp16", 5, False), (80, 160, "fp16", 7, True), (96, 192, "bf16", 160, False), (112, 240, "bf16", 9, True), (64, 208, "fp16", 33, True)]


@pytest.mark.parametrize("m,n,dtype,tokens,pack", WIDE)
def test_against_oracle(m, n, dtype, tokens, pack):
    x, left, right = make_inputs(tokens, m * n, dtype, 7 * m + n + tokens, True, mn=(m, n))
    sample = slice(None) if tokens <= 40 else torch.linspace(0, tokens - 1, 40).long()
    ref_codes, ref_scales = O.flatquant_quantize(t2f(x[sample]), t2f(left), t2f(right), 0.9, pack, dtype)
    codes, scales = abi_quantize(x.to(DEV), left.to(DEV), right.to(DEV), 0.9, pack, dtype, policy=2)
    assert lib.qo_last_quantizer_path() == 2 and lib.qo_device_status(stream_ptr()) == N.QO_OK
    check(codes.cpu()[sample].numpy(), t2f(scales)[sample if isinstance(sample, slice) else sample.numpy()], ref_codes, ref_scales, pack)


# row counts that a pair's MMAs (32 rows a step, half from each CTA) pad, and columns of the second CTA from one quadrant to four;
# a pair with one token, two pairs, one pair more than the device has, and pairs with uneven shares
PAIR = [(48, 176, "bf16", 2, True), (80, 144, "fp16", 75, True), (112, 256, "bf16", 149, False), (16, 192, "bf16", 74, True), (96, 224, "fp16", 3, True)]


@pytest.mark.parametrize("m,n,dtype,tokens,pack", PAIR)
def test_cta_pairs_against_oracle(m, n, dtype, tokens, pack):
    test_against_oracle(m, n, dtype, tokens, pack)


def test_transform_only_and_dispatch():
    x, left, right = make_inputs(6, 128 * 224, "bf16", 3, True)
    ref = O.kronecker_transform(t2f(x), t2f(left), t2f(right), "bf16").reshape(6, -1)
    z = torch.empty(6, 128 * 224, device=DEV)
    xd, ld, rd = x.to(DEV), left.to(DEV), right.to(DEV)
    N.check(lib.qo_flatquant_transform(ptr(xd), 128 * 224, ptr(ld), ptr(rd), ptr(z), 6, 128, 224, QD["bf16"], stream_ptr()))
    torch.cuda.synchronize()
    assert lib.qo_last_quantizer_path() == 2
    # a sum next to a rounding boundary of Y or Z may round to the neighbour (2^-8 relative in bf16)
    err = (z.cpu() - torch.from_numpy(ref)).abs()
    assert (err > 2.0 ** -7 * torch.from_numpy(ref).abs() + 2.0 ** -7 * float(abs(ref).mean())).float().mean() == 0
    abi_quantize(xd, ld, rd, 0.9, True, "bf16")
    assert lib.qo_last_quantizer_path() == 2


@pytest.mark.parametrize("dtype", ["bf16", "fp16"])
@pytest.mark.parametrize("pack", [True, False])
def test_special_tokens_equal_the_simt_kernel(dtype, pack):
    m, n = 32, 160
    x, left, right = make_inputs(12, m * n, dtype, 5, True, mn=(m, n))
    x[1, 77] = float("inf")
    x[2, 5000] = -float("inf")
    x[3, 0] = float("nan")
    x[4] = float("nan")
    x[5] = 0.0
    x[6] = 1e-7  # fp16: subnormal values and scale (the codes depend on the order of the sums, hence the scale only)
    x[7, 3], x[7, 4000] = float("inf"), float("inf")
    got = abi_quantize(x.to(DEV), left.to(DEV), right.to(DEV), 0.9, pack, dtype, policy=2)
    ref = abi_quantize(x.to(DEV), left.to(DEV), right.to(DEV), 0.9, pack, dtype, policy=1)
    special = torch.tensor([1, 2, 3, 4, 5, 7], device=DEV)
    assert torch.equal(got[0][special], ref[0][special])
    assert torch.equal(got[1][special], ref[1][special])
    assert torch.allclose(got[1][6], ref[1][6], rtol=2.0 ** -7)


@pytest.mark.parametrize("dtype,clip", [("bf16", 0.9), ("bf16", 1e6), ("fp16", 1.0), ("fp16", 1.3), ("fp16", 1e6)])
@pytest.mark.parametrize("pack", [True, False])
def test_scales_over_the_whole_range_of_the_type(dtype, clip, pack):
    """Identity transforms, so that every kernel quantizes the same values: from the smallest to the largest scales, and
    infinite ones (the row's largest value times the clip ratio leaves the type), the codes are those of the SIMT kernel."""
    m, n = 32, 160
    g = torch.Generator().manual_seed(11)
    z = torch.randn(64, m * n, dtype=torch.float64, generator=g).clamp_(-1.99, 1.99)
    low, high = (-130, 126) if dtype == "bf16" else (-23, 15)
    x = (z * torch.exp2(torch.linspace(low, high, 64).round().double())[:, None]).to(TD[dtype]).to(DEV)
    assert bool(x.isfinite().all())
    left, right = torch.eye(m, dtype=x.dtype, device=DEV), torch.eye(n, dtype=x.dtype, device=DEV)
    got = abi_quantize(x, left, right, clip, pack, dtype, policy=2)
    ref = abi_quantize(x, left, right, clip, pack, dtype, policy=1)
    assert bool(ref[1].isinf().any()) == (clip > 1)
    assert torch.equal(got[1], ref[1]) and torch.equal(got[0], ref[0])


@pytest.mark.parametrize("mode,shift", [("packed", 4), ("int8", 1), ("transform", 4)])
def test_outputs_off_a_16_byte_boundary(mode, shift):
    """The C entry points take outputs of these widths at any boundary of their element type, on the SIMT kernel."""
    m, n, tokens = 16, 160, 9
    x, left, right = (t.to(DEV) for t in make_inputs(tokens, m * n, "bf16", 8, True, mn=(m, n)))
    size = tokens * m * n * {"packed": 1, "int8": 2, "transform": 8}[mode] // 2
    results = []
    for policy, at in ((1, 0), (0, shift)):
        raw = torch.full((size + 32,), 77, dtype=torch.uint8, device=DEV)
        scales = torch.zeros(tokens, device=DEV)
        out = C.c_void_p(raw.data_ptr() + at)
        N.check(lib.qo_set_kernel_policy(policy))
        try:
            if mode == "transform":
                N.check(lib.qo_flatquant_transform(ptr(x), m * n, ptr(left), ptr(right), out, tokens, m, n, QD["bf16"], stream_ptr()))
            else:
                N.check(lib.qo_flatquant_quantize(ptr(x), m * n, ptr(left), ptr(right), out, ptr(scales), tokens, m, n, 0.9, QD["bf16"],
                                                  int(mode == "packed"), QD["fp32"], stream_ptr()))
        finally:
            lib.qo_set_kernel_policy(0)
        torch.cuda.synchronize()
        assert lib.qo_last_quantizer_path() == 1
        assert bool((raw[:at] == 77).all()) and bool((raw[at + size:] == 77).all())
        results.append((raw[at:at + size].clone(), scales))
    assert torch.equal(results[0][0], results[1][0]) and torch.equal(results[0][1], results[1][1])


@pytest.mark.parametrize("pack", [True, False])
def test_a_scale_that_rounds_to_zero(pack):
    """fp16 tokens of up to three subnormal steps: three steps over 7 round to a scale of 0, and the quotients' limits are the
    codes: 7, -8, and 0 for 0.  Identity transforms keep the values."""
    m, n = 32, 160
    g = torch.Generator().manual_seed(3)
    x = (torch.randint(-3, 4, (6, m * n), generator=g) * 2.0 ** -24).half().to(DEV)
    left, right = torch.eye(m, dtype=x.dtype, device=DEV), torch.eye(n, dtype=x.dtype, device=DEV)
    codes, scales = abi_quantize(x, left, right, 1.0, pack, "fp16", policy=2)
    assert bool((scales == 0).all())
    if pack:
        codes = ((codes[:, :, None] >> (4 * torch.arange(8, dtype=torch.int32, device=DEV))) & 15).reshape(6, m * n) - 8
    assert torch.equal(codes.int(), torch.where(x > 0, 7, torch.where(x < 0, -8, 0)).int())


def test_a_token_has_the_same_codes_alone_and_in_a_batch():
    """Rows are independent: one token, three and all of them give the same bits."""
    x, left, right = (t.to(DEV) for t in make_inputs(64, 128 * 224, "bf16", 17, True, mn=(128, 224)))
    codes, scales = abi_quantize(x, left, right, 0.9, True, "bf16")
    for size in (1, 3):
        for i in range(0, 64 - size + 1, size):
            c, s = abi_quantize(x[i:i + size], left, right, 0.9, True, "bf16")
            assert torch.equal(c, codes[i:i + size]) and torch.equal(s, scales[i:i + size])

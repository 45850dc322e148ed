"""The GEMM that unpacks inside the kernel, with K split over clusters of CTA pairs and with the weights in the [K/8, N] layout:
accumulators and outputs are the bits of the kernels that multiply widened operands (policy 3) at the edges of its tiles."""
import pytest
import torch

import quant_ops_b200 as q
from helpers import N, abi_int4_matmul, launched_kernels, lib, make_inputs, stream_ptr

pytestmark = pytest.mark.gpu
DEV = "cuda:0"

# rows: one, around a CTA's and a pair's rows; columns: one tile, ragged tiles, as many as leave four to one slices of K;
# K: the shortest that are split, odd numbers of stages, a single stage and three of them unsplit at prefill sizes, and three shapes
# whose K of less than 2048 keeps them on widened operands
SHAPES = [(1, 4096, 4096), (33, 256, 256), (100, 1024, 264), (128, 2048, 1024), (129, 2304, 1000), (256, 14336, 4096), (257, 4096, 4096),
          (300, 2816, 520), (512, 1280, 4096), (200, 4096, 14336), (333, 4096, 14328), (700, 11008, 4088), (1030, 4096, 1024),
          (33, 2048, 256), (100, 2304, 264), (1536, 256, 2048), (1500, 768, 2056)]


def problem(t, k, n, seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    words = lambda *s: torch.randint(-2 ** 31, 2 ** 31, s, dtype=torch.int64, device=DEV, generator=g).to(torch.int32)
    return words(t, k // 8), words(n, k // 8), torch.rand(t, device=DEV, generator=g) + 0.01, torch.rand(n, device=DEV, generator=g) * 1e-4


@pytest.mark.parametrize("t,k,n", SHAPES)
@pytest.mark.parametrize("layout", ["weights_t_view", "reference_contiguous"])
def test_same_bits_as_the_widening_path(t, k, n, layout):
    a, w, sa, sb = problem(t, k, n, t + k + n)
    b = w.t() if layout == "weights_t_view" else w.t().contiguous()
    for out_dtype in ("fp16", "bf16"):
        ref, ref_acc = abi_int4_matmul(a, b, sa, sb, out_dtype, True, policy=3)
        before = lib.qo_kernel_launch_count()
        got, acc = abi_int4_matmul(a, b, sa, sb, out_dtype, True, policy=2)
        assert (lib.qo_kernel_launch_count() - before == 1) == (k >= 2048 or t >= 1500)  # one launch: no widening pass
        assert lib.qo_device_status(stream_ptr()) == N.QO_OK
        assert torch.equal(acc, ref_acc)
        assert torch.equal(got.view(torch.int16), ref.view(torch.int16))


@pytest.mark.parametrize("t,n", [(4, 1288), (40, 1280), (40, 1288), (300, 1024), (1024, 3072)])
@pytest.mark.parametrize("k", [131072 - 256, 131072])
def test_extreme_codes_of_the_longest_reductions(t, n, k):
    """Zeroed operands are codes of -8 on both sides.  With the factor 256 of the kernels that keep the nibbles in the high
    half of a byte the sum is 2^31 at K = 131072, one more than an int32 holds: those kernels take the shorter products only
    (few rows, split K, prefill), and longer ones run on widened operands."""
    a, w = torch.zeros(t, k // 8, dtype=torch.int32, device=DEV), torch.zeros(n, k // 8, dtype=torch.int32, device=DEV)
    sa, sb = torch.full((t,), 2.0 ** -10, device=DEV), torch.ones(n, device=DEV)
    for b in (w.t(), w.t().contiguous()):
        before = lib.qo_kernel_launch_count()
        out, acc = abi_int4_matmul(a, b, sa, sb, "fp16", True)
        assert (lib.qo_kernel_launch_count() - before == 1) == (k < 131072)  # one launch: no widening pass
        assert int(acc.min()) == int(acc.max()) == 64 * k
        assert float(out.min()) == float(out.max()) == 64 * k / 1024


def test_row_strides_and_repeated_calls():
    a, w, sa, sb = problem(150, 4096, 2048, 9)
    wide = torch.zeros(150, 516, dtype=torch.int32, device=DEV)
    wide[:, :512] = a
    cols = torch.zeros(512, 2056, dtype=torch.int32, device=DEV)
    cols[:, :2048] = w.t()
    ref = abi_int4_matmul(a, w.t(), sa, sb, "bf16", policy=3)
    for _ in range(30):  # the rings are reused as exchange buffers: a leftover of one call must not reach the next
        assert torch.equal(abi_int4_matmul(wide[:, :512], cols[:, :2048], sa, sb, "bf16"), ref)
        assert torch.equal(abi_int4_matmul(a, w.t(), sa, sb, "bf16"), ref)


@pytest.mark.parametrize("tokens,k,n_out", [(33, 4096, 4096), (64, 14336, 4096), (256, 14336, 4096), (130, 4096, 11008)])
def test_layer_with_early_weight_loads(tokens, k, n_out):
    """Inside the layer the first weight stages are requested before the quantizer ahead has finished: the same bits as the
    two calls by hand, with bias, call after call."""
    x, left, right = make_inputs(tokens, k, "bf16", tokens + n_out, True)
    xd, ld, rd = x.to(DEV), left.to(DEV), right.to(DEV)
    _, w, _, sb = problem(1, k, n_out, 4)
    bias = torch.randn(n_out, device=DEV).bfloat16()
    codes, scales = q.flatquant_dynamic_quantize(xd, ld, rd, 0.9, True)
    want = (q.int4_matmul_ex(codes, w.t(), scales, sb, torch.bfloat16).float() + bias.float()).bfloat16()
    for _ in range(10):
        assert torch.equal(q.w4a4_linear(xd, ld, rd, w, sb, bias, 0.9), want)
    q.device_status()


# few column tiles and a long K run on widened operands; either side of each line
FEW_TILES = [("layer", 96, 4096, 256, True), ("layer", 97, 4096, 256, False), ("layer", 128, 4096, 1024, False), ("layer", 128, 4096, 1032, True),
             ("layer", 128, 3072, 256, True), ("layer", 129, 4096, 1024, True), ("layer", 128, 6144, 1024, True), ("layer", 64, 8192, 512, False),
             ("layer", 64, 8192, 520, True), ("layer", 256, 8192, 256, False), ("layer", 257, 8192, 256, True), ("rows", 128, 4096, 256, False), ("rows", 128, 4096, 264, True), ("rows", 128, 8192, 1024, False),
             ("rows", 128, 7168, 1024, True), ("rows", 96, 8192, 768, True), ("rows", 40, 14336, 512, False), ("columns", 128, 8192, 512, False),
             ("columns", 96, 8192, 512, True), ("columns", 20, 14336, 256, False), ("columns", 20, 14336, 264, True)]


@pytest.mark.parametrize("form,t,k,n,unpacks", FEW_TILES)
def test_route_and_bits_at_the_lines(form, t, k, n, unpacks):
    a, w, sa, sb = problem(t, k, n, t + k + n)
    if form == "layer":
        x, left, right = (v.to(DEV) for v in make_inputs(t, k, "bf16", t + n, True))
        codes, scales = q.flatquant_dynamic_quantize(x, left, right, 0.9, True)
        want = q.int4_matmul_ex(codes, w.t(), scales, sb, torch.bfloat16)
        call = lambda: q.w4a4_linear(x, left, right, w, sb, None, 0.9)
    else:
        b = w.t() if form == "rows" else w.t().contiguous()
        want = abi_int4_matmul(a, b, sa, sb, "fp16", policy=3)
        call = lambda: q.int4_matmul(a, b, sa, sb)
    assert torch.equal(call(), want)
    names = launched_kernels(call)
    assert any("gemm_s4_unpack_kernel" in name for name in names) == unpacks
    assert any("widen" in name for name in names) != unpacks


# layers that keep an int8 copy of their weights: packed weights where the unpacking kernel is the faster one, else the copy
KEPT = [(128, 4096, 2048, False), (129, 4096, 2048, True), (160, 4096, 11008, True), (257, 4096, 11008, False), (1024, 4096, 1024, False),
        (1040, 4096, 1024, True), (384, 8192, 1024, False), (400, 8192, 1024, True), (256, 8192, 1792, False), (300, 8192, 4352, False), (600, 8192, 3072, False), (520, 8192, 2816, True),
        (900, 8192, 3072, True), (600, 2048, 1024, True), (256, 1024, 1024, False)]


@pytest.mark.parametrize("t,k,n,packed", KEPT)
def test_route_and_bits_with_kept_weights(t, k, n, packed):
    _, w, _, sb = problem(1, k, n, t + n)
    x, left, right = (v.to(DEV) for v in make_inputs(t, k, "bf16", t + n, True))
    kept = q.prepare_weights(w)
    codes, scales = q.flatquant_dynamic_quantize(x, left, right, 0.9, True)
    call = lambda: q.w4a4_linear_prepared(x, left, right, w, kept, sb, None, 0.9)
    assert torch.equal(call(), abi_int4_matmul(codes, w.t(), scales, sb, "bf16", policy=3))
    names = launched_kernels(call)
    assert len(names) == 2 and any("gemm_s4_unpack_kernel" in name for name in names) == packed

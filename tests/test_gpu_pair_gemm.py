"""The CTA-pair GEMM (calls of more than 512 rows, dense weights from 65 rows on) at the sizes where it can go wrong: ragged token tiles and segments, empty
segments, out-features that are odd multiples of 128, cut tiles of the last wave, one to many K-chunks.  Small-integer
activations make every product and sum exact, so the comparison with a plain f32 matmul is exact; the GELU form is compared
with the one-CTA kernel bit for bit."""
import pytest
import torch

from jarvis_b200 import _lib, ops

pytestmark = pytest.mark.gpu


def _weights(G, N, K, gen, prepared):
    w = torch.randint(-1, 2, (G, N, K), generator=gen, device="cuda").float()
    packed = torch.stack([ops.pack_codes(w[g]) for g in range(G)])
    return w, ops.prepare_weights(packed) if prepared else packed


@pytest.mark.parametrize("M,N,K,prepared", [(513, 128, 256, True), (767, 384, 256, False), (1024, 1024, 1024, True),
                                            (2331, 3072, 1024, True), (9473, 1024, 512, False), (19000, 256, 2048, True)])
def test_single_matrix_forms_are_exact(M, N, K, prepared):
    gen = torch.Generator(device="cuda").manual_seed(M)
    x = torch.randint(-3, 4, (M, K), generator=gen, device="cuda").bfloat16()
    w, packed = _weights(1, N, K, gen, prepared)
    alpha = torch.tensor([0.25], device="cuda")
    want = 0.25 * (x.float() @ w[0].t())                          # integers below 2^24 times a power of two
    got = ops.ternary_linear(x, packed[0], alpha, epilogue=ops.EPI_F32, prepared=prepared)
    assert torch.equal(got, want)
    assert torch.equal(ops.ternary_linear(x, packed[0], alpha, prepared=prepared), want.bfloat16())
    base = torch.randint(-8, 9, (M, N), generator=gen, device="cuda").float()
    assert torch.equal(ops.ternary_linear(x, packed[0], alpha, epilogue=ops.EPI_RESID_F32, out=base.clone(), prepared=prepared), base + want)
    a = ops.ternary_linear(x, packed[0], alpha, epilogue=ops.EPI_GELU_BF16, prepared=prepared)
    b = ops.ternary_linear(x, packed[0], alpha, epilogue=ops.EPI_GELU_BF16, prepared=prepared, token_tile=128)
    assert torch.equal(a, b)
    assert _lib.device_status() == 0


@pytest.mark.parametrize("M,N,K,cuts", [(513, 128, 256, [0, 0, 513, 513, 513]), (1500, 384, 512, [0, 1, 257, 900, 1500]),
                                        (4662, 2048, 1024, [0, 1100, 2400, 3600, 4662]), (20000, 1024, 256, [0, 10000, 10001, 19999, 20000])])
def test_grouped_forms_are_exact(M, N, K, cuts):
    gen = torch.Generator(device="cuda").manual_seed(M)
    x = torch.randint(-3, 4, (M, K), generator=gen, device="cuda").bfloat16()
    w, packed = _weights(4, N, K, gen, True)
    alpha = torch.tensor([0.25, 0.5, 1.0, 2.0], device="cuda")
    offs = torch.tensor(cuts, dtype=torch.int32, device="cuda")
    want = torch.cat([float(alpha[g]) * (x[cuts[g]:cuts[g + 1]].float() @ w[g].t()) for g in range(4)])
    assert torch.equal(ops.ternary_linear_grouped(x, packed, alpha, offs, epilogue=ops.EPI_F32, prepared=True), want)
    assert torch.equal(ops.ternary_linear_grouped(x, packed, alpha, offs, prepared=True), want.bfloat16())
    out = want.clone()
    assert torch.equal(ops.ternary_linear_grouped(x, packed, alpha, offs, epilogue=ops.EPI_RESID_F32, out=out, prepared=True), 2 * want)
    assert _lib.device_status() == 0


@pytest.mark.parametrize("M,N,K", [(1, 128, 256), (33, 640, 1024), (64, 50304, 1024), (65, 128, 256), (100, 640, 1024),
                                   (256, 50304, 1024), (257, 384, 512), (513, 128, 256), (1111, 640, 1024), (3000, 50304, 256)])
def test_dense_weights_are_exact(M, N, K):
    gen = torch.Generator(device="cuda").manual_seed(N)
    x = torch.randint(-3, 4, (M, K), generator=gen, device="cuda").bfloat16()
    w = torch.randint(-3, 4, (N, K), generator=gen, device="cuda").bfloat16()
    want = x.float() @ w.float().t()
    assert torch.equal(ops.dense_linear(x, w, out_dtype=torch.float32), want)
    assert torch.equal(ops.dense_linear(x, w), want.bfloat16())
    assert _lib.device_status() == 0


@pytest.mark.parametrize("M,N,K", [(65, 128, 256), (513, 384, 256), (767, 1024, 1024)])
def test_outputs_that_start_on_a_16_byte_boundary(M, N, K):
    """The entry points take them; the CTA-pair kernel's stores need 32 bytes."""
    gen = torch.Generator(device="cuda").manual_seed(M)
    x = torch.randint(-3, 4, (M, K), generator=gen, device="cuda").bfloat16()
    w, packed = _weights(1, N, K, gen, True)
    alpha = torch.tensor([0.25], device="cuda")
    want = 0.25 * (x.float() @ w[0].t())
    dense = 0.25 * w[0].bfloat16()

    def out(dtype):
        t = torch.zeros(M * N + 32, dtype=dtype, device="cuda")
        at = 16 // t.element_size() if t.data_ptr() % 32 == 0 else 0
        t = t[at:at + M * N].view(M, N)
        assert t.data_ptr() % 32 == 16
        return t
    offs = torch.tensor([0, M], dtype=torch.int32, device="cuda")
    f32, bf16 = torch.float32, torch.bfloat16
    assert torch.equal(ops.ternary_linear(x, packed[0], alpha, epilogue=ops.EPI_F32, out=out(f32), prepared=True), want)
    assert torch.equal(ops.ternary_linear(x, packed[0], alpha, out=out(bf16), prepared=True), want.bfloat16())
    assert torch.equal(ops.ternary_linear(x, packed[0], alpha, epilogue=ops.EPI_RESID_F32, out=out(f32), prepared=True), want)
    assert torch.equal(ops.ternary_linear_grouped(x, packed, alpha, offs, out=out(bf16), prepared=True), want.bfloat16())
    assert torch.equal(ops.dense_linear(x, dense, out_dtype=f32, out=out(f32)), want)
    assert torch.equal(ops.dense_linear(x, dense, out=out(bf16)), want.bfloat16())
    gelu = ops.ternary_linear(x, packed[0], alpha, epilogue=ops.EPI_GELU_BF16, out=out(bf16), prepared=True)
    assert torch.equal(gelu, ops.ternary_linear(x, packed[0], alpha, epilogue=ops.EPI_GELU_BF16, prepared=True))
    assert _lib.device_status() == 0


@pytest.mark.parametrize("M,cut", [(40, (0, 33)), (300, (5, 170)), (513, (0, 500)), (1500, (3, 1025))])
def test_residual_of_one_segment_leaves_the_rows_around_it(M, cut):
    gen = torch.Generator(device="cuda").manual_seed(M)
    x = torch.randint(-3, 4, (M, 256), generator=gen, device="cuda").bfloat16()
    w, packed = _weights(1, 384, 256, gen, True)
    offs = torch.tensor(cut, dtype=torch.int32, device="cuda")
    base = torch.randint(-8, 9, (M, 384), generator=gen, device="cuda").float()
    want = base.clone()
    want[cut[0]:cut[1]] += 0.5 * (x[cut[0]:cut[1]].float() @ w[0].t())
    got = ops.ternary_linear_grouped(x, packed, torch.tensor([0.5], device="cuda"), offs, epilogue=ops.EPI_RESID_F32, out=base.clone(),
                                     prepared=True)
    assert torch.equal(got, want)
    assert _lib.device_status() == 0

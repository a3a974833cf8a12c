"""bf16 products whose contraction is shared by several CTA pairs (`bf16_splits` in csrc/bindings.cpp): fp32 slabs summed in order."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# the LM head's input gradient at two row counts; a last share that is shorter than the others; rows and columns outside whole tiles, the
# result a slice of a wider matrix; just long enough for two shares and just too short
@pytest.mark.parametrize("m,n,k", [(1024, 768, 50304), (3840, 768, 8192), (200, 104, 6152), (33, 8, 2048), (64, 264, 2112), (64, 264, 1984)])
@pytest.mark.parametrize("b_mn", [False, True])
def test_shared_contraction(m, n, k, b_mn):
    from gpt_moe_b200.ops import cuda_ops
    torch.manual_seed(8)
    c = cuda_ops.ext()
    a = torch.randn(m, k, device="cuda").bfloat16()
    b = torch.randn((k, n) if b_mn else (n, k), device="cuda").bfloat16()
    wide = torch.full((m + 1, n + 24), 5.0, device="cuda", dtype=torch.bfloat16)
    c.gemm_bf16(a, b, wide[:m, 8: 8 + n], False, b_mn, 0.25)
    want = 0.25 * (a.double() @ (b.double() if b_mn else b.double().t()))
    # one rounding to bf16 (2^-9 relative at most) over sums that are fp32
    assert ((wide[:m, 8: 8 + n].double() - want).abs() <= 2 ** -8 * want.abs() + 1e-5 * k ** 0.5).all()
    assert (wide[m] == 5).all() and (wide[:, :8] == 5).all() and (wide[:, 8 + n:] == 5).all()
    again = torch.empty(m, n, device="cuda", dtype=torch.bfloat16)
    c.gemm_bf16(a, b, again, False, b_mn, 0.25)
    assert torch.equal(again, wide[:m, 8: 8 + n])                  # the shares are summed in the same order every time
    cuda_ops.check_status()


@pytest.mark.parametrize("m,n,k", [(64, 264, 8192), (64, 264, 64)])          # shared by several pairs, and whole
@pytest.mark.parametrize("offset", [1, 2, 4])
def test_an_output_off_the_16_byte_grid_is_refused(m, n, k, offset):
    """Before any launch: the sum over the shares stores 8 bytes at a time."""
    from gpt_moe_b200.ops import cuda_ops
    a, b = torch.zeros(m, k, device="cuda").bfloat16(), torch.zeros(n, k, device="cuda").bfloat16()
    wide = torch.full((m, n + 8), 5.0, device="cuda", dtype=torch.bfloat16)
    with pytest.raises(RuntimeError, match="16-byte"):
        cuda_ops.ext().gemm_bf16(a, b, wide[:, offset: offset + n])
    assert (wide == 5).all()
    cuda_ops.check_status()


def test_contractions_that_a_sum_would_not_repay_stay_whole():
    """us, whole / the best of 2 to 8 shares: 360 x 1024 x 2048 12 / 14, 1536 x 768 x 3072 16 / 18, 2048 x 1024 x 4096 20 / 23; the others gain."""
    from gpt_moe_b200.ops import cuda_ops
    splits = cuda_ops.ext().bf16_splits
    for m, n, k in ((360, 1024, 2048), (1536, 768, 3072), (2048, 1024, 4096)):
        assert splits(m, n, k, True, 148) == 1
    for m, n, k, narrow in ((360, 768, 8192, True), (1024, 768, 50304, True), (2048, 768, 50304, True), (9472, 768, 50304, False)):
        assert splits(m, n, k, narrow, 148) > 1


# where shares begin: few columns with long enough a contraction; a last share shorter than the others; rows of several tiles
@pytest.mark.parametrize("m,n,k", [(64, 264, 4096), (300, 520, 5000), (33, 8, 4160), (1100, 264, 9000)])
@pytest.mark.parametrize("b_mn", [False, True])
def test_shared_contractions_at_the_line(m, n, k, b_mn):
    from gpt_moe_b200.ops import cuda_ops
    torch.manual_seed(9)
    c = cuda_ops.ext()
    assert c.bf16_splits(m, n, k, n > 128, 148) > 1
    a = torch.randn(m, k, device="cuda").bfloat16()
    b = torch.randn((k, n) if b_mn else (n, k), device="cuda").bfloat16()
    wide = torch.full((m + 1, n + 24), 5.0, device="cuda", dtype=torch.bfloat16)
    c.gemm_bf16(a, b, wide[:m, 8: 8 + n], False, b_mn)
    want = a.double() @ (b.double() if b_mn else b.double().t())
    assert ((wide[:m, 8: 8 + n].double() - want).abs() <= 2 ** -8 * want.abs() + 1e-5 * k ** 0.5).all()      # as above
    assert (wide[m] == 5).all() and (wide[:, :8] == 5).all() and (wide[:, 8 + n:] == 5).all()
    cuda_ops.check_status()


# contractions that an fp32 result would share: the addend comes in once, also on top of what the output holds.  Whole numbers below 2^24: every order
# of the sums gives the same
@pytest.mark.parametrize("m,n,k,b_mn", [(638, 48, 8192, False), (767, 128, 4096, True), (1062, 864, 1296, True)])
@pytest.mark.parametrize("accumulate", [False, True])
def test_an_addend_beside_an_fp32_result_is_added_once(m, n, k, b_mn, accumulate):
    from gpt_moe_b200.ops import cuda_ops
    torch.manual_seed(15)
    a = torch.randint(-1, 2, (m, k), device="cuda").bfloat16()
    b = torch.randint(-1, 2, (k, n) if b_mn else (n, k), device="cuda").bfloat16()
    c = 2 * torch.randint(-60, 60, (m, n), device="cuda").bfloat16()
    d = torch.randint(-1000, 1000, (m, n), device="cuda").float()
    want = a.double() @ (b.double() if b_mn else b.double().t()) - 0.5 * c.double() + (d.double() if accumulate else 0)
    cuda_ops.ext().gemm_bf16(a, b, d, False, b_mn, 1.0, -0.5, c, accumulate)
    assert torch.equal(d.double(), want)
    cuda_ops.check_status()

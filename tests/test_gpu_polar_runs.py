"""Polar Express on the small side (`polar_express` in csrc/bindings.cpp): runs of steps and single steps against 64 bits."""
import pytest
import torch

from gpt_moe_b200.ops import reference as ref

pytestmark = pytest.mark.gpu


def _exact(g):
    x = g.double()
    x = x / (x.norm(dim=(-2, -1), keepdim=True) * 1.02 + 1e-6)
    for a, b, c in ref.POLAR_EXPRESS_COEFFS:
        gram = x @ x.mT
        x = a * x + (b * gram + c * (gram @ gram)) @ x
    return x


def _error(x, exact):
    return ((x.double() - exact).norm(dim=(-2, -1)) / exact.norm(dim=(-2, -1))).max().item()


# (batch, rows, columns): runs with whole tiles, with ragged ones, at the least height, just too few tiles for runs, just too narrow for them
# (single steps with the fp16 Gram matrices); few rows (one launch): every height, as wide as high, more matrices than SMs
@pytest.mark.parametrize("shape", [(16, 768, 1536), (12, 520, 2056), (64, 256, 704), (8, 256, 768), (16, 768, 1528), (3, 8, 768),
                                   (4, 32, 1536), (2, 24, 264), (150, 16, 16)])
@pytest.mark.parametrize("spectrum", ["gaussian", "decaying"])
def test_polar_express_is_no_further_from_64_bits_than_single_steps_in_bf16(shape, spectrum):
    from gpt_moe_b200.ops import cuda_ops
    torch.manual_seed(9)
    n, m, k = shape
    g = torch.randn(n, m, k, device="cuda")
    if spectrum == "decaying":
        u, v = torch.linalg.qr(torch.randn(n, m, m, device="cuda"))[0], torch.linalg.qr(torch.randn(n, k, m, device="cuda"))[0]
        g = (u * torch.exp(-12 * torch.arange(1, m + 1, device="cuda") / m)) @ v.mT
    raw = (g * 3e-4).bfloat16()
    sumsq = raw.float().pow(2).sum(dim=(-2, -1))
    exact = _exact(raw)
    got = cuda_ops.polar_express_bf16(raw.clone(), sumsq)
    assert got.dtype == torch.bfloat16 and got.shape == raw.shape
    # the same steps one by one with every matrix rounded to bf16; a tenth for the luck of single roundings, and 2^-8 for the output's own
    plain = _error(ref.polar_express(raw, dtype=torch.bfloat16), exact)
    assert _error(got, exact) < 1.1 * plain + 2 ** -8
    normalised = (raw.double() / (raw.double().norm(dim=(-2, -1), keepdim=True) * 1.02 + 1e-6)).bfloat16()
    assert _error(cuda_ops.polar_express_bf16(normalised.clone()), _exact(normalised * 1.0)) < 1.1 * plain + 2 ** -6
    cuda_ops.check_status()


# runs of steps, single steps, and the kernel for few rows
@pytest.mark.parametrize("shape", [(16, 768, 1536), (8, 256, 768), (3, 512, 512), (4, 32, 768)])
@pytest.mark.parametrize("weak", [1e-4, 1e-5, 1e-6, 1e-7])
def test_rows_far_below_the_others_keep_their_direction(shape, weak):
    """A 2-norm over the matrix does not see them: the error is taken over the weak rows alone."""
    from gpt_moe_b200.ops import cuda_ops
    torch.manual_seed(10)
    n, m, k = shape
    g = torch.randn(n, m, k, device="cuda")
    rows = torch.arange(m, device="cuda") % 8 == 3
    g[:, rows] *= weak
    raw = g.bfloat16()
    exact = _exact(raw)
    got = cuda_ops.polar_express_bf16(raw.clone(), raw.float().pow(2).sum(dim=(-2, -1)))
    plain = ref.polar_express(raw, dtype=torch.bfloat16)
    for part in (rows, ~rows):            # bounds as above
        assert _error(got[:, part], exact[:, part]) < 1.1 * _error(plain[:, part], exact[:, part]) + 2 ** -8
    cuda_ops.check_status()


@pytest.mark.parametrize("shape", [(16, 768, 1536), (3, 512, 512), (4, 32, 768)])
@pytest.mark.parametrize("norm", [1e-9, 1e-11, 1e-13])
def test_matrices_that_are_nearly_zero_keep_their_direction(shape, norm):
    """The momentum of an expert that has seen no token for long: 1 / (1.02 norm + 1e-6) no longer brings its norm to one."""
    from gpt_moe_b200.ops import cuda_ops
    torch.manual_seed(11)
    g = torch.randn(shape, device="cuda")
    raw = (g * (norm / g.norm(dim=(-2, -1), keepdim=True))).bfloat16()
    exact = _exact(raw)
    got = cuda_ops.polar_express_bf16(raw.clone(), raw.float().pow(2).sum(dim=(-2, -1)))
    assert _error(got, exact) < 1.1 * _error(ref.polar_express(raw, dtype=torch.bfloat16), exact) + 2 ** -8
    cuda_ops.check_status()


# runs, single steps, few rows in one launch, and more rows than columns
@pytest.mark.parametrize("shape", [(16, 768, 1536), (3, 512, 520), (4, 16, 264), (2, 264, 136)])
def test_matrices_with_a_pitch_of_their_own(shape):
    from gpt_moe_b200.ops import cuda_ops
    torch.manual_seed(12)
    n, m, k = shape
    wide = torch.randn(n, m + 2, k + 24, device="cuda").bfloat16()
    x = wide[:, 1: m + 1, 8: k + 8]
    sumsq = x.float().pow(2).sum(dim=(-2, -1))
    assert torch.equal(cuda_ops.polar_express_bf16(x, sumsq), cuda_ops.polar_express_bf16(x.contiguous(), sumsq))
    exact = _exact(x)
    plain = _error(ref.polar_express(x, dtype=torch.bfloat16), exact)
    assert _error(cuda_ops.polar_express_bf16(x, sumsq), exact) < 1.1 * plain + 2 ** -8
    cuda_ops.check_status()

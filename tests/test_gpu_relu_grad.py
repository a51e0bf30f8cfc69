"""A training layer's backward with an upstream gradient at any address: the
kernels want 16-byte alignment, a caller's contiguous BF16 view need not have
it (a slice of a flat buffer of several layers' gradients)."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("no CUDA device", allow_module_level=True)

from hmfem_b200 import guess  # noqa: E402


@pytest.mark.parametrize("relu", [True, False])
@pytest.mark.parametrize("offset", [0, 1, 4, 7])
def test_backward_takes_a_gradient_at_any_address(offset, relu):
    dims, n = (9, 7, 5), 9 * 7 * 5
    gen = torch.Generator().manual_seed(offset)
    x = torch.randn(2, n, 8, generator=gen).bfloat16().cuda().requires_grad_()
    w = (0.1 * torch.randn(27, 16, 16, generator=gen)).cuda().requires_grad_()
    b = torch.randn(16, generator=gen).cuda().requires_grad_()
    # small integers: every sum below 2^8 per channel and cell is exact
    flat = torch.randint(-2, 3, (16 * n + 8,), generator=gen).bfloat16().cuda()
    up = flat[offset:offset + 16 * n].view(2, n, 8)
    assert up.is_contiguous() and up.data_ptr() % 16 == (2 * offset) % 16
    got = torch.autograd.grad(guess.conv(x, w, b, dims, relu=relu), (x, w, b), up)
    ref = torch.autograd.grad(guess.conv(x, w, b, dims, relu=relu), (x, w, b), up.clone())
    guess.check_errors()
    assert torch.equal(got[0], ref[0]) and torch.equal(got[2], ref[2])
    # (the weight gradient's atomic sums have no fixed order)
    assert float((got[1] - ref[1]).abs().max()) <= 1e-5 * float(ref[1].abs().max())

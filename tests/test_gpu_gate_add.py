"""x + gate * y in one kernel against the fp64 value rounded once to BF16 (the product of two BF16 values
is exact in fp32, so fp32 addition followed by the BF16 rounding is what torch.addcmul computes)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch,rows,n,offset,sliced", [
    (1, 1, 8, 0, False), (2, 33, 1152, 0, True), (3, 7, 2056, 0, True), (2, 5, 4096, 0, False),
    (2, 5, 1156, 0, False),        # n off 16 bytes: torch's path
    (2, 5, 64, 1, False),          # a base off 16 bytes: torch's path
])
def test_equals_addcmul_bit_for_bit(sdk, batch, rows, n, offset, sliced):
    from slidesparse_diffusion_b200 import backend
    sdk.load_native()
    gen = torch.Generator(device="cuda").manual_seed(n + rows)
    def make(*shape):
        flat = torch.randn(torch.Size(shape).numel() + offset, generator=gen, device="cuda").to(torch.bfloat16)
        return flat[offset:].view(shape)
    x, y = make(batch, rows, n), make(batch, rows, n)
    gate = make(batch, 3 * n)[:, n:2 * n] if sliced else make(batch, n)
    x.view(-1)[::5], y.view(-1)[::7] = 0, float("inf")
    got = torch.ops.slidesparse_b200.gate_add(x, gate, y)
    expect = torch.addcmul(x, gate[:, None], y)
    assert torch.equal(got.isnan(), expect.isnan())
    assert torch.equal(got.nan_to_num().view(torch.int16), expect.nan_to_num().view(torch.int16))
    assert torch.equal(backend.gate_add(x, gate, y).nan_to_num(), expect.nan_to_num())


def test_differentiates_through_torch(sdk):
    from slidesparse_diffusion_b200 import backend
    sdk.load_native()
    x, y = (torch.randn(2, 4, 64, device="cuda", dtype=torch.bfloat16, requires_grad=True) for _ in range(2))
    backend.gate_add(x, torch.ones(2, 64, device="cuda", dtype=torch.bfloat16), y).sum().backward()
    assert torch.equal(x.grad, torch.ones_like(x)) and torch.equal(y.grad, torch.ones_like(y))

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


def _operands(batch=2, rows=5, n=64):
    gen = torch.Generator(device="cuda").manual_seed(3)
    make = lambda *shape: torch.randn(*shape, generator=gen, device="cuda").to(torch.bfloat16)
    return (make(batch, rows, n), make(batch, n), make(batch, rows, n)), (make(batch, rows, n), make(batch, n), make(batch, rows, n))


def _entries():
    from slidesparse_diffusion_b200 import backend, denoiser
    return backend.gate_add, denoiser.gate, torch.ops.slidesparse_b200.gate_add


def test_forward_mode_derivatives_are_those_of_addcmul(sdk):
    """Dual tensors do not require gradients; each operand on its own and all together carry a tangent."""
    sdk.load_native()
    fwd = torch.autograd.forward_ad
    reference = lambda x, gate, y: torch.addcmul(x, gate[:, None], y)
    values, tangents = _operands()
    for entry in _entries():
        for dual in ((0,), (1,), (2,), (0, 1, 2)):
            with fwd.dual_level():
                operands = [fwd.make_dual(v, t) if i in dual else v for i, (v, t) in enumerate(zip(values, tangents))]
                got, expect = fwd.unpack_dual(entry(*operands)), fwd.unpack_dual(reference(*operands))
                assert got.tangent is not None and torch.equal(got.tangent, expect.tangent)
                assert torch.equal(got.primal, expect.primal)
        got, expect = torch.func.jvp(entry, values, tangents), torch.func.jvp(reference, values, tangents)
        assert torch.equal(got[0], expect[0]) and torch.equal(got[1], expect[1])


def test_gradients_and_batches_under_function_transforms(sdk, recwarn):
    sdk.load_native()
    reference = lambda x, gate, y: torch.addcmul(x, gate[:, None], y)
    values, tangents = _operands()
    pairs = [torch.stack(p) for p in zip(values, tangents)]
    for entry in _entries():
        for wanted in range(3):
            loss = lambda f: torch.func.grad(lambda *a: f(*a).float().square().sum(), argnums=wanted)(*values)
            assert torch.equal(loss(entry), loss(reference))
        for dims in ((0, 0, 0), (0, None, 0), (None, 0, None)):
            operands = [p if d == 0 else p[0] for p, d in zip(pairs, dims)]
            assert torch.equal(torch.vmap(entry, dims)(*operands), torch.vmap(reference, dims)(*operands))
        leaves = [v.clone().requires_grad_() for v in values]
        entry(*leaves).sum().backward()
        assert torch.equal(leaves[1].grad, values[2].sum(1))
    assert not [w for w in recwarn if "vmap" in str(w.message) or "batching" in str(w.message)]

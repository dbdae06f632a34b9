"""Kernels whose launches overlap (programmatic stream serialization) on buffers that each of them writes
for the next: the same bits as with the overlap switched off, over many links and reused memory."""
import pytest
import torch

from gpu_util import option

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
LINKS = 24


def _packed(k, n, mode, seed):
    from slidesparse_diffusion_b200 import routing
    gen = torch.Generator(device=DEV).manual_seed(seed)
    layer = torch.nn.Linear(k, n, device=DEV, dtype=torch.bfloat16).requires_grad_(False)
    layer.weight.normal_(0, 0.05, generator=gen)
    layer.bias.normal_(0, 0.1, generator=gen)
    return routing.pack_members([layer], mode)


@pytest.mark.parametrize("rows,mode", [(32, 4), (352, 6), (2048, 8)])
def test_gated_norm_and_gate_add_chain(sdk, backend, rows, mode):
    """FFN-out added to the residual in place -> norm and modulation of that residual -> its projection as
    the next update, added by the gate kernel."""
    batch, hidden, wide = 2, 384, 768
    down, up = _packed(wide, hidden, mode, 1), _packed(hidden, hidden + wide, mode, 2)
    gen = torch.Generator(device=DEV).manual_seed(rows)
    make = lambda *shape: torch.randn(*shape, generator=gen, device=DEV).to(torch.bfloat16) * 0.5
    start, first = make(batch, rows, hidden), make(batch, rows, wide)
    shift, scale, gate = make(batch, hidden), make(batch, hidden), make(batch, hidden)

    def chain():
        residual, branch, out = start.clone(), first.clone(), []
        for _ in range(LINKS):
            down.forward_fused(branch, backend.Prologue.gelu(), gate=gate, residual=residual)
            both = up.forward_fused(residual, backend.Prologue.norm_modulate(shift, scale))
            out.append(residual.clone())
            residual = backend.gate_add(residual, gate, both[..., :hidden].contiguous())
            residual.mul_(0.5)
            again = up.forward_fused(backend.gate_add(residual, gate, out[-1]), backend.Prologue.norm_modulate(shift, scale))
            branch.copy_(again[..., hidden:])
        return torch.stack(out + [residual])

    overlapped = [chain() for _ in range(4)]
    with option(backend, "pdl", 0):
        expect = chain()
    assert expect.isfinite().all() and backend.device_status() == 0
    for got in overlapped:
        assert torch.equal(got, expect)


@pytest.mark.parametrize("width", [77, 192])
def test_projection_of_a_projection(sdk, backend, width):
    """Output of one projection straight into the next, by 16-byte and by 2-byte loads and stores."""
    there, back = _packed(width, 328, 6, 3), _packed(328, width, 6, 4)
    x = torch.randn(160, width, generator=torch.Generator(device=DEV).manual_seed(5), device=DEV).to(torch.bfloat16)

    def chain():
        y = x
        for _ in range(LINKS):
            y = back(there(y), output_addend=y)
        return y

    overlapped = [chain() for _ in range(4)]
    with option(backend, "pdl", 0):
        expect = chain()
    for got in overlapped:
        assert torch.equal(got, expect)
    assert backend.device_status() == 0

"""The addend epilogues of the GEMM at the edges of their dispatch: 16-byte aligned rows (staged tiles and
TMA stores) and rows that are not, token tiles that end in a half chunk, one row, one 8-channel group.
Every output bit is compared with the CPU oracle; the columns beside the output must stay untouched."""
import numpy as np
import pytest
import torch

from gpu_util import bits, check, option, prepare_case, ptr, stream

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("m,n,offset,tile", [(1, 8, 8, 0), (33, 264, 8, 128), (500, 776, 16, 240), (257, 520, 0, 256),
                                             (33, 264, 1, 0), (257, 77, 8, 0), (1000, 3072, 24, 240)])
def test_addend_alignments_and_tiles(backend, oracle, oracle_c, m, n, offset, tile):
    k, mode = 768, 6
    case = prepare_case(oracle, m, k, n, mode, seed=m + n)
    dev = lambda a, dtype=None: torch.from_numpy(np.ascontiguousarray(a)).to(DEV)
    gen = torch.Generator().manual_seed(m)
    wide = torch.randn(m, n + 40, generator=gen).to(torch.bfloat16)
    wide_dev = wide.to(DEV)
    addend = wide_dev[:, offset:offset + n]
    out = torch.full((m, n + 24), 7.0, dtype=torch.bfloat16, device=DEV)
    q, packed, meta = dev(case["q"]), dev(case["packed"]), dev(case["meta_b200"].view(np.int32))
    sa, sw, bias = dev(case["sa"]), dev(case["scales"]), dev(case["bias"])
    with option(backend, "token_tile", tile):
        check(backend, backend.library().ss_gemm_run(
            ptr(q), ptr(packed), ptr(meta), ptr(sa), ptr(sw), ptr(bias), ptr(addend), addend.stride(0), ptr(out), out.stride(0),
            m, n, q.shape[0], packed.shape[0], q.shape[1], stream()))
    torch.cuda.synchronize()
    expect = oracle_c.epilogue(case["acc"], case["sa"], case["scales"], case["bias"], bits(wide[:, offset:offset + n]))
    got = bits(out)
    assert np.array_equal(got[:, :n], expect)
    assert (got[:, n:] == bits(torch.tensor([7.0]).to(torch.bfloat16))[0]).all()
    assert backend.device_status() == 0

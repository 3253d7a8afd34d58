"""act_quant where it changes from one block per half-warp to four: the rows of a tensor on either side of the line equal those of its parts."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("extra", [-1, 0, 1, 64])
@pytest.mark.parametrize("fmt", [None, "ue8m0"])
def test_rows_do_not_depend_on_their_number(extra, fmt):
    import kernel
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    rows = sms * 16 * 10 + extra                      # blocks of 128 at which the launch changes
    g = torch.Generator(device="cuda").manual_seed(rows)
    x = torch.randn(rows, 128, generator=g, device="cuda", dtype=torch.float32).bfloat16()
    q, s = kernel.act_quant(x, 128, fmt)
    parts = [kernel.act_quant(p.contiguous(), 128, fmt) for p in (x[:15], x[15:rows // 3], x[rows // 3:])]
    assert torch.equal(q.view(torch.uint8), torch.cat([p[0].view(torch.uint8) for p in parts]))
    assert torch.equal(s, torch.cat([p[1] for p in parts]))

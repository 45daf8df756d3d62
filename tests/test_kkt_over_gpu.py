"""The preparation whose K tile lies where the chunks' areas are (calls that keep neither A nor w, without norms): several items per CTA,
with and without a second chunk, one and several heads each.  The raw forward, whose preparation keeps its K tile, gives the same bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("lens, hk, hv", [
    # 592 CTAs are resident: 225 pairs of chunks x 4 and x 8 heads, pairs of one chunk beside pairs of two; 700 pairs of one chunk;
    # 593 pairs of one head: one CTA has a second item
    ([5000, 63, 64, 130, 9000, 1, 127, 128, 8192, 65, 5313], 4, 4),
    ([5000, 63, 64, 130, 9000, 1, 127, 128, 8192, 65, 5313], 8, 32),
    ([64, 1, 33, 64, 7] * 140, 1, 3),
    ([593 * 128], 1, 1),
    ([593 * 128 - 65], 1, 1),
])
def test_bits_of_the_raw_forward(lens, hk, hv, dtype):
    import flashqla_b200 as fq
    pairs = sum(-(-n // 128) for n in lens)
    resident = 4 * torch.cuda.get_device_properties(0).multi_processor_count
    assert pairs * hk > resident or resident != 592, "every CTA has one item: the K tile is not loaded a second time"
    gen = torch.Generator(device="cuda").manual_seed(len(lens) + hv)
    T = sum(lens)
    q, k, v = (torch.randn(1, T, n, 128, generator=gen, device="cuda") for n in (hk, hk, hv))
    q, k = (torch.nn.functional.normalize(x, dim=-1).to(dtype) for x in (q, k))
    g = torch.nn.functional.logsigmoid(torch.randn(1, T, hv, generator=gen, device="cuda"))
    beta = torch.sigmoid(torch.randn(1, T, hv, generator=gen, device="cuda"))
    cu = torch.tensor([0] + lens).cumsum(0).int().cuda()
    raw = fq.chunk_gated_delta_rule_fwd(q, k, v.to(dtype), g, beta, cu_seqlens=cu)
    for _ in range(3):
        with torch.no_grad():
            o, final = fq.chunk_gated_delta_rule(q, k, v.to(dtype), g, beta, output_final_state=True, cu_seqlens=cu)
        fq.check_device_status()
        assert torch.equal(o, raw[2]) and torch.equal(final, raw[4])

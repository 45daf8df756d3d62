"""Order in which the reverse scan starts the sequences of a packed batch: longest first, which is what the segment planner reckons with
when it leaves a batch uncut (``cp.plan_segments``), and without influence on the gradients."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lens", [[70, 1, 500, 64, 129, 0, 300], [33, 2000, 64]])
def test_longest_first(lens, monkeypatch):
    from flashqla_b200 import _cabi, chunk
    Hk, Hv, T = 2, 4, sum(lens)
    gen = torch.Generator(device="cuda").manual_seed(len(lens))
    q, k = (torch.nn.functional.normalize(torch.randn(1, T, Hk, 128, generator=gen, device="cuda"), dim=-1).bfloat16() for _ in range(2))
    v, do = (torch.randn(1, T, Hv, 128, generator=gen, device="cuda").bfloat16() for _ in range(2))
    g = torch.nn.functional.logsigmoid(torch.randn(1, T, Hv, generator=gen, device="cuda"))
    beta = torch.rand(1, T, Hv, generator=gen, device="cuda")
    h0 = 0.1 * torch.randn(len(lens), Hv, 128, 128, generator=gen, device="cuda")
    cu = torch.tensor([0] + lens).cumsum(0).int().cuda()
    fwd = chunk.chunk_gated_delta_rule_fwd(q, k, v, g, beta, initial_state=h0, cu_seqlens=cu, output_h=True, output_v_new=True,
                                           auto_cp=False)
    orders, host = [], _cabi.host()

    class Recorder:
        def __getattr__(self, name):
            return getattr(host, name)

        def chunk_bwd(self, *args):
            given = args[11]
            results = [host.chunk_bwd(*args[:11], order, *args[12:]) for order in (given, None, given.flip(0).contiguous())]
            orders.append(given)
            for other in results[1:]:
                assert all(torch.equal(a, b) for a, b in zip(results[0], other))
            return results[0]

    monkeypatch.setattr(_cabi, "host", lambda: Recorder())
    chunk.chunk_gated_delta_rule_bwd(q, k, v, fwd[0], beta, fwd[1], do, dht=0.1 * torch.ones_like(h0), initial_state=h0, cu_seqlens=cu,
                                     h=fwd[3], v_new=fwd[5], auto_cp=False)
    assert [lens[i] for i in orders[0].tolist()] == sorted(lens, reverse=True)

"""Height of the recurrent kernel's tiles: 16 rows while all tiles are resident at once, 32 beyond.  Batches on either side of the
line (four to six tiles per SM) against the oracle."""
import pytest
import torch

from oracle import gdr_oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [73, 74, 75, 92, 93, 111, 112, 147, 148, 149])
@pytest.mark.parametrize("pool_dtype", [torch.float32, torch.bfloat16])
def test_decode_around_the_line(n, pool_dtype):
    import flashqla_b200 as fq
    gen = torch.Generator().manual_seed(n)
    q, k, v = (torch.randn(1, n, 1, 128, generator=gen).bfloat16() for _ in range(3))
    a, b = torch.randn(1, n, 1, generator=gen), torch.randn(1, n, 1, generator=gen)
    A_log, dt = torch.zeros(1), torch.zeros(1)
    state = (0.1 * torch.randn(n, 1, 128, 128, generator=gen)).to(pool_dtype)
    pool = state.cuda()
    o = fq.fused_sigmoid_gating_delta_rule_update(A_log.cuda(), a.cuda(), dt.cuda(), q.cuda(), k.cuda(), v.cuda(), b.cuda(), pool,
                                                  use_qk_l2norm_in_kernel=True)
    ref_state = state.float()
    ref = orc.recurrent_update_ref(A_log, a, dt, q, k, v, b, ref_state, use_qk_l2norm=True)
    # fp32 arithmetic, one rounding of o (2^-9 of values up to 1) and of a bf16 state
    assert orc.max_abs(o.float().cpu(), ref) <= 3e-3
    assert orc.max_abs(pool.float().cpu(), ref_state) <= (1e-4 if pool_dtype == torch.float32 else 2.0 ** -8)

"""The recurrent op's kernels for one step, for a chain of steps and for everything else give the same bits: where a call goes (number
of steps, cached states, heads) must not show in its results."""
import pytest
import torch

from oracle import gdr_oracle as orc

pytestmark = pytest.mark.gpu


def inputs(n, steps, hk, hv, dtype, seed, l2norm):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    length = 1.0 if l2norm else 0.08  # of sqrt(128): keys as they are may not be longer than about 1
    q, k = ((length * torch.randn(1, n * steps, hk, 128, generator=gen, device="cuda")).to(dtype) for _ in range(2))
    v = torch.randn(1, n * steps, hv, 128, generator=gen, device="cuda").to(dtype)
    a, b = (torch.randn(1, n * steps, hv, generator=gen, device="cuda") for _ in range(2))
    A_log, dt = torch.randn(hv, generator=gen, device="cuda"), torch.randn(hv, generator=gen, device="cuda")
    pool = 0.1 * torch.randn(n + 2, hv, 128, 128, generator=gen, device="cuda")
    slots = torch.randperm(n + 2, generator=gen, device="cuda")[:n].int()
    return A_log, a, dt, q, k, v, b, pool, slots


# a block of steps is four; the chain kernel has all but the call of 148 heads, with 16 rows up to 18 heads; its 32-row tiles are
# all resident up to 185, and from 186 on its CTAs have a second item
@pytest.mark.parametrize("l2norm", [False, True])
@pytest.mark.parametrize("n, steps, hk, hv, dtype", [
    (1, 2, 1, 1, torch.bfloat16), (3, 3, 2, 4, torch.float16), (148, 4, 1, 1, torch.bfloat16), (149, 5, 1, 1, torch.bfloat16),
    (186, 8, 1, 1, torch.bfloat16), (7, 9, 4, 32, torch.bfloat16), (47, 33, 1, 8, torch.float16)])
def test_chain_equals_the_general_kernel(n, steps, hk, hv, dtype, l2norm):
    """States cached in 16 bits (the kernel for chains) are the rounded values of those cached in fp32 (the general one); o, and a
    pool that is updated (no cache: chains, too), are the same bits; and both stand at the oracle."""
    import flashqla_b200 as fq
    A_log, a, dt, q, k, v, b, pool, slots = inputs(n, steps, hk, hv, dtype, n + steps, l2norm)

    def call(cached, state_pool, **kw):
        if cached is not None:
            kw.update(intermediate_states_buffer=cached, intermediate_state_indices=torch.arange(n, dtype=torch.int32, device="cuda"))
        return fq.fused_sigmoid_gating_delta_rule_update(A_log, a, dt, q, k, v, b, state_pool, slots, use_qk_l2norm_in_kernel=l2norm, **kw)

    c32 = torch.zeros(n, steps, hv, 128, 128, device="cuda")
    c16 = torch.zeros(n, steps, hv, 128, 128, dtype=torch.bfloat16, device="cuda")
    pools = [pool.clone() for _ in range(3)]
    o32, o16, o0 = call(c32, pools[0]), call(c16, pools[1]), call(None, pools[2])
    fq.check_device_status()
    assert torch.equal(o32, o16) and torch.equal(o32, o0)
    assert torch.equal(c32.bfloat16(), c16)
    assert torch.equal(pools[0], pools[1]) and torch.equal(pools[0], pools[2])
    if n * hv > 300 or steps > 9:
        return
    ref_pool = pool.cpu().clone()
    ref = orc.recurrent_update_ref(A_log.cpu(), a.cpu(), dt.cpu(), q.cpu(), k.cpu(), v.cpu(), b.cpu(), ref_pool, slots.cpu().long(),
                                   use_qk_l2norm=l2norm)
    # fp32 arithmetic over up to nine steps; o is rounded once (bf16: 2^-9 of its values)
    assert orc.max_abs(o16.float().cpu(), ref) <= 2.0 ** -8 * max(ref.abs().max().item(), 1.0)
    assert orc.max_abs(pools[1].cpu(), ref_pool) <= 1e-4 * max(ref_pool.abs().max().item(), 1.0)


@pytest.mark.parametrize("pool_dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("l2norm", [False, True])
def test_one_step_on_either_side_of_the_line(pool_dtype, l2norm):
    """1024 fp32 heads go to the kernel for one step, 1056 to the general one (bf16 pools: both to the former): what the first 32
    sequences get does not depend on it.  cu_seqlens of single tokens, which the general kernel takes, give the same as well."""
    import flashqla_b200 as fq
    A_log, a, dt, q, k, v, b, pool, _ = inputs(33, 1, 16, 32, torch.bfloat16, 1, l2norm)
    pool, slots = pool.to(pool_dtype), torch.arange(33, dtype=torch.int32, device="cuda")
    got = []
    for n, cu in ((32, False), (33, False), (32, True)):
        p = pool.clone()
        kw = dict(cu_seqlens=torch.arange(n + 1, dtype=torch.int32, device="cuda")) if cu else {}
        o = fq.fused_sigmoid_gating_delta_rule_update(A_log, a[:, :n].contiguous(), dt, q[:, :n].contiguous(), k[:, :n].contiguous(),
                                                      v[:, :n].contiguous(), b[:, :n].contiguous(), p, slots[:n],
                                                      use_qk_l2norm_in_kernel=l2norm, **kw)
        got.append((o[:, :32], p[:32]))
    fq.check_device_status()
    for o, p in got[1:]:
        assert torch.equal(o, got[0][0]) and torch.equal(p, got[0][1])

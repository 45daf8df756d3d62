"""Which of the recurrent op's kernels a call gets and the height of its tiles, 16 or 32 rows: both follow from how many tiles there are
per SM.  Batches on either side of the lines against the oracle, and against each other bit by bit."""
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


def names_of(call):
    """Names of the recurrent kernels that ``call`` launches, and what it returns."""
    from torch.profiler import ProfilerActivity, profile
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        got = call()
        torch.cuda.synchronize()
    return [e.name for e in prof.events() if "recurrent" in e.name], got


# both sides of every line between the two kernels and the two tile heights
@pytest.mark.parametrize("n, steps, cached, kernel, rows", [
    (18, 4, True, "chain", 16), (19, 4, True, "chain", 32), (37, 5, True, "general", 16), (38, 5, True, "general", 32), (38, 8, True, "chain", 32),
    (74, 6, True, "general", 32), (75, 6, True, "chain", 32), (92, 8, True, "chain", 32), (93, 8, True, "general", 32),
    (132, 6, True, "general", 32), (148, 2, True, "general", 32), (149, 2, True, "chain", 32), (185, 8, True, "chain", 32),
    (200, 5, True, "general", 32), (288, 4, True, "general", 32), (300, 4, True, "chain", 32), (300, 8, True, "general", 32),
    (512, 5, True, "chain", 32), (4, 64, False, "general", 16), (80, 9, False, "chain", 32), (112, 4, False, "general", 32), (264, 6, False, "general", 32)])
def test_chains_on_either_side_of_their_lines(n, steps, cached, kernel, rows):
    """Several steps, cached in bf16 or not at all: which kernel and tile height a call gets depends on its heads and steps, its bits do not."""
    import flashqla_b200 as fq
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("the lines depend on the number of SMs")
    gen = torch.Generator(device="cuda").manual_seed(n + steps)
    q, k, v = (torch.randn(1, n * steps, 1, 128, generator=gen, device="cuda").bfloat16() for _ in range(3))
    a, b = (torch.randn(1, n * steps, 1, generator=gen, device="cuda") for _ in range(2))
    pool = 0.1 * torch.randn(n, 1, 128, 128, generator=gen, device="cuda")
    zero, slots = torch.zeros(1, device="cuda"), torch.arange(n, dtype=torch.int32, device="cuda")

    def call(block_dv, ragged=False):
        state, scratch = pool.clone(), torch.zeros(n, steps, 1, 128, 128, dtype=torch.bfloat16, device="cuda") if cached else None
        kw = dict(intermediate_states_buffer=scratch, intermediate_state_indices=slots) if cached else {}
        if ragged:  # (always the general kernel)
            kw["cu_seqlens"] = steps * torch.arange(n + 1, dtype=torch.int32, device="cuda")
        o = fq.fused_sigmoid_gating_delta_rule_update(zero, a, zero, q, k, v, b, state, slots, block_dv=block_dv, **kw)
        return [o, state] + ([scratch] if cached else [])

    names, got = names_of(lambda: call(None))
    expected = f"recurrent_chain_kernel<__nv_bfloat16, {'__nv_bfloat16' if cached else 'float'}, float, {rows // 16}>" if kernel == "chain" else \
        f"recurrent_kernel<__nv_bfloat16, {'__nv_bfloat16' if cached else 'float'}, float, {rows // 16}, false>"
    assert len(names) == 1 and expected in names[0], names
    for other in (call(16), call(32), call(None, ragged=True)):
        assert all(torch.equal(x, y) for x, y in zip(got, other))
    fq.check_device_status()


@pytest.mark.parametrize("pool_dtype, n, kernel, rows", [
    (torch.float32, 1, "step", 16), (torch.float32, 64, "step", 16), (torch.float32, 65, "step", 32), (torch.float32, 92, "step", 32),
    (torch.float32, 93, "step", 16), (torch.float32, 129, "step", 16), (torch.float32, 130, "general", 32), (torch.float32, 148, "general", 32),
    (torch.float32, 149, "step", 32), (torch.float32, 246, "step", 32), (torch.float32, 247, "general", 32), (torch.float32, 296, "general", 32),
    (torch.float32, 297, "step", 32), (torch.float32, 1024, "step", 32), (torch.float32, 1025, "general", 32),
    (torch.bfloat16, 74, "general", 16), (torch.bfloat16, 148, "general", 32), (torch.bfloat16, 149, "step", 32), (torch.bfloat16, 246, "step", 32),
    (torch.bfloat16, 247, "general", 32), (torch.bfloat16, 296, "general", 32), (torch.bfloat16, 297, "step", 32), (torch.bfloat16, 1025, "step", 32)])
def test_one_step_on_either_side_of_its_lines(pool_dtype, n, kernel, rows):
    """One token per sequence: which kernel and tile height a call gets depends on its heads and its pool, its bits do not; with and
    without a cached state of either type, q, k, v of either type, against single tokens by cu_seqlens, which the general kernel takes."""
    import flashqla_b200 as fq
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("the lines depend on the number of SMs")
    gen = torch.Generator(device="cuda").manual_seed(n)
    zero, slots = torch.zeros(1, device="cuda"), torch.arange(n, dtype=torch.int32, device="cuda")
    a, b = (torch.randn(1, n, 1, generator=gen, device="cuda") for _ in range(2))
    pool = (0.1 * torch.randn(n, 1, 128, 128, generator=gen, device="cuda")).to(pool_dtype)
    for dtype, cache in ((torch.bfloat16, None), (torch.float16, torch.float32), (torch.bfloat16, torch.bfloat16)):
        q, k, v = (torch.randn(1, n, 1, 128, generator=gen, device="cuda").to(dtype) for _ in range(3))

        def call(block_dv, ragged=False):
            state, scratch = pool.clone(), torch.zeros(n, 1, 1, 128, 128, dtype=cache or torch.float32, device="cuda")
            kw = dict(intermediate_states_buffer=scratch, intermediate_state_indices=slots) if cache else {}
            if ragged:
                kw["cu_seqlens"] = torch.arange(n + 1, dtype=torch.int32, device="cuda")
            o = fq.fused_sigmoid_gating_delta_rule_update(zero, a, zero, q, k, v, b, state, slots, block_dv=block_dv, **kw)
            return o, state, scratch

        names, got = names_of(lambda: call(None))
        types = ", ".join({torch.bfloat16: "__nv_bfloat16", torch.float16: "__half", torch.float32: "float"}[t]
                          for t in (dtype, torch.bfloat16 if cache == torch.bfloat16 else torch.float32, pool_dtype))
        expected = f"recurrent_step_kernel<{types}, {rows // 16}>" if kernel == "step" else f"recurrent_kernel<{types}, {rows // 16}, false>"
        assert len(names) == 1 and expected in names[0], names
        for other in (call(16), call(32), call(None, ragged=True)):
            assert all(torch.equal(x, y) for x, y in zip(got, other))
    fq.check_device_status()


@pytest.mark.parametrize("n, rows", [(74, 16), (75, 32), (111, 32), (138, 32), (139, 16), (148, 16), (149, 32)])
def test_trees_with_fp32_scratch(n, rows):
    """32-row tiles of a tree are resident three per SM: with 139 to 148 heads two rounds of 16 rows take less time.  Either height
    gives the same bits."""
    import flashqla_b200 as fq
    from torch.profiler import ProfilerActivity, profile
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("the line depends on the number of SMs")
    gen = torch.Generator().manual_seed(n)
    q, k, v = (torch.randn(1, 3 * n, 1, 128, generator=gen).bfloat16().cuda() for _ in range(3))
    a, b = (torch.randn(1, 3 * n, 1, generator=gen).cuda() for _ in range(2))
    pool = (0.1 * torch.randn(n, 1, 128, 128, generator=gen)).cuda()
    parents = torch.tensor([[-1, 0, 0]] * n, dtype=torch.int32, device="cuda")

    def step(block_dv):
        scratch = torch.zeros(n, 3, 1, 128, 128, device="cuda")
        o = fq.fused_sigmoid_gating_delta_rule_update(
            torch.zeros(1, device="cuda"), a, torch.zeros(1, device="cuda"), q, k, v, b, pool, torch.arange(n, dtype=torch.int32, device="cuda"),
            use_qk_l2norm_in_kernel=True, disable_state_update=True, intermediate_states_buffer=scratch,
            intermediate_state_indices=torch.arange(n, dtype=torch.int32, device="cuda"), retrieve_parent_token=parents, block_dv=block_dv)
        return o, scratch

    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        got = step(None)
        torch.cuda.synchronize()
    names = [e.name for e in prof.events() if "recurrent_kernel" in e.name]
    assert names and all(f", {rows // 16}, true>" in name for name in names), names
    for other in (step(16), step(32)):
        assert torch.equal(got[0], other[0]) and torch.equal(got[1], other[1])

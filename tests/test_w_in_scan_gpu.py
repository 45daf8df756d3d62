"""Calls that keep no ``w`` (inference): the scan forms ``w`` itself, of the same operands in the same
order, so that the results are those of the raw forward, which the other files hold to the oracle, bit by bit."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def inputs(lens, Hk, Hv, dtype, weak, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    T = sum(lens)
    q, k, v = (torch.randn(1, T, n, 128, generator=gen, device="cuda") for n in (Hk, Hk, Hv))
    q, k = (torch.nn.functional.normalize(x, dim=-1) for x in (q, k))
    g = torch.nn.functional.logsigmoid(torch.randn(1, T, Hv, generator=gen, device="cuda"))
    if weak:  # heads that hardly ever forget: transition matrices of the segments
        g = g / 64
        g[..., 0] = 0
    beta = torch.sigmoid(torch.randn(1, T, Hv, generator=gen, device="cuda"))
    h0 = 0.1 * torch.randn(len(lens) + 3, Hv, 128, 128, generator=gen, device="cuda")
    cu = torch.tensor([0] + list(lens)).cumsum(0).int().cuda()
    return q.to(dtype), k.to(dtype), v.to(dtype), g, beta, h0, cu


CASES = [  # lengths, heads, weak gates
    ([1], (1, 1), False),
    ([130, 64], (2, 4), True),
    ([65536 // 8 + 1], (4, 8), False),                     # segments, warm-up inside the scan
    ([65536 // 4 + 37], (2, 4), True),                     # segments, state-only passes and transition matrices
    ([1, 63, 64, 65, 127, 128, 129, 192, 193, 2048, 777], (16, 32), False),
    ([3] * 500 + [641], (8, 32), True),                    # one chunk each: the rings turn over with every sequence
]


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("lens, heads, weak", CASES)
def test_op(lens, heads, weak, dtype):
    import flashqla_b200 as fq
    q, k, v, g, beta, h0, cu = inputs(lens, *heads, dtype, weak, 3)
    h0 = h0[:len(lens)]
    raw = fq.chunk_gated_delta_rule_fwd(q, k, v, g, beta, initial_state=h0, cu_seqlens=cu)
    with torch.no_grad():
        o, final = fq.chunk_gated_delta_rule(q, k, v, g, beta, initial_state=h0, output_final_state=True, cu_seqlens=cu)
    fq.check_device_status()
    assert torch.equal(o, raw[2]) and torch.equal(final, raw[4])
    with torch.no_grad():
        again = fq.chunk_gated_delta_rule(q, k, v, g, beta, initial_state=h0, output_final_state=True, cu_seqlens=cu)
    assert torch.equal(o, again[0]) and torch.equal(final, again[1])


@pytest.mark.parametrize("pool_dtype, norm", [(torch.float32, True), (torch.bfloat16, False)])
@pytest.mark.parametrize("lens, heads, weak", CASES)
def test_pool(lens, heads, weak, pool_dtype, norm):
    import flashqla_b200 as fq
    q, k, v, g, beta, h0, cu = inputs(lens, *heads, torch.bfloat16, weak, 4)
    slots = torch.randperm(len(h0), device="cuda")[:len(lens)].int()
    if len(lens) > 1:
        slots[0] = -1  # no slot: from zero, nothing written
    gate = dict(out_norm_gate=torch.randn_like(v), out_norm_weight=torch.rand(128, device="cuda") + 0.5) if norm else {}
    pools = [h0.to(pool_dtype).clone() for _ in range(2)]
    raw = fq.chunk_gated_delta_rule_fwd(
        3 * q, 2 * k, v, g, beta, initial_state=pools[0], initial_state_indices=slots, final_state_out=pools[0],
        final_state_indices=slots, cu_seqlens=cu, transpose_state_layout=True, use_qk_l2norm_in_kernel=True, **gate)
    o, _ = fq.prefill_into_state_pool(3 * q, 2 * k, v, g, beta, pools[1], slots, cu_seqlens=cu, continue_from_pool=True,
                                      use_qk_l2norm_in_kernel=True, **gate)
    fq.check_device_status()
    assert torch.equal(o, raw[2]) and torch.equal(pools[1], pools[0])
    rest = torch.ones(len(h0), dtype=torch.bool, device="cuda")
    used = slots[slots >= 0].long()
    rest[used] = False
    assert torch.equal(pools[1][rest], h0.to(pool_dtype)[rest])
    assert not any(torch.equal(pools[1][slot], h0.to(pool_dtype)[slot]) for slot in used)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("lens, heads, weak", CASES[1:5])
def test_layer_call(lens, heads, weak, dtype):
    """Raw gates and beta logits in the activation type, into a pool of either type."""
    import flashqla_b200 as fq
    q, k, v, g, _, h0, cu = inputs(lens, *heads, dtype, weak, 7)
    slots = torch.randperm(len(h0), device="cuda")[:len(lens)].int()
    kw = dict(A_log=torch.rand(heads[1], device="cuda").log() - (3 if weak else 0), dt_bias=torch.randn(heads[1], device="cuda"),
              beta_is_logit=True, use_qk_l2norm_in_kernel=True)
    a, b = torch.randn_like(g).to(dtype), 3 * torch.randn_like(g).to(dtype)
    for pool_dtype in (torch.float32, torch.bfloat16):
        pools = [h0.to(pool_dtype).clone() for _ in range(2)]
        raw = fq.chunk_gated_delta_rule_fwd(5 * q, k / 3, v, a, b, initial_state=pools[0], initial_state_indices=slots,
                                            final_state_out=pools[0], final_state_indices=slots, cu_seqlens=cu,
                                            transpose_state_layout=True, **kw)
        o, _ = fq.prefill_into_state_pool(5 * q, k / 3, v, a, b, pools[1], slots, cu_seqlens=cu, continue_from_pool=True, **kw)
        fq.check_device_status()
        assert torch.isfinite(o.float()).all() and torch.equal(o, raw[2]) and torch.equal(pools[1], pools[0])


@pytest.mark.parametrize("B, T, heads", [(1, 64, (1, 1)), (3, 200, (2, 4)), (5, 1500, (4, 4))])
@pytest.mark.parametrize("transposed", [False, True])
def test_equal_lengths_and_betas_of_either_sign(B, T, heads, transposed):
    import flashqla_b200 as fq
    gen = torch.Generator(device="cuda").manual_seed(T)
    q, k, v = (torch.randn(B, T, n, 128, generator=gen, device="cuda") for n in (heads[0], heads[0], heads[1]))
    q, k = (torch.nn.functional.normalize(x, dim=-1) for x in (q, k))
    q, k, v = q.bfloat16(), k.bfloat16(), v.bfloat16()
    g = torch.nn.functional.logsigmoid(torch.randn(B, T, heads[1], generator=gen, device="cuda"))
    beta = 2 * torch.rand(B, T, heads[1], generator=gen, device="cuda") - 1
    beta[:, ::5] = 0
    h0 = 0.1 * torch.randn(B, heads[1], 128, 128, generator=gen, device="cuda")
    raw = fq.chunk_gated_delta_rule_fwd(q, k, v, g, beta, initial_state=h0, transpose_state_layout=transposed)
    with torch.no_grad():
        o, final = fq.chunk_gated_delta_rule(q, k, v, g, beta, initial_state=h0, output_final_state=True,
                                             transpose_state_layout=transposed)
    with_grad, _ = fq.chunk_gated_delta_rule(q, k, v, g, beta.clone().requires_grad_(), initial_state=h0, output_final_state=True,
                                             transpose_state_layout=transposed)
    fq.check_device_status()
    assert torch.equal(o, raw[2]) and torch.equal(final, raw[4]) and torch.equal(o, with_grad.detach())


def test_trace_is_filled():
    """A trace buffer that is set records calls that keep nothing, too, and changes no result."""
    import flashqla_b200 as fq
    from flashqla_b200 import _cabi
    q, k, v, g, beta, _, cu = inputs([64 * 12], 1, 2, torch.bfloat16, False, 6)
    with torch.no_grad():
        plain = fq.chunk_gated_delta_rule(q, k, v, g, beta, output_final_state=True, cu_seqlens=cu)
        buf = torch.zeros(3 * 4 * 16 + 3 * 2, dtype=torch.int64, device="cuda")  # roles x chunks x events, then the two CTAs
        _cabi.check(_cabi.lib().qla_set_trace_buffer(buf.data_ptr(), buf.numel()), "qla_set_trace_buffer")
        try:
            traced = fq.chunk_gated_delta_rule(q, k, v, g, beta, output_final_state=True, cu_seqlens=cu)
            torch.cuda.synchronize()
        finally:
            _cabi.check(_cabi.lib().qla_set_trace_buffer(None, 0), "qla_set_trace_buffer")
    fq.check_device_status()
    assert torch.equal(plain[0], traced[0]) and torch.equal(plain[1], traced[1])
    phases, ctas = buf[:192].view(3, 4, 16), buf[192:].view(2, 3)
    assert (phases[0, :, [0, 2, 3, 4, 6, 7, 8, 9, 10, 11]] > 0).all() and (phases[1, :, 2:6] > 0).all() and (phases[2, :, [6, 8, 9, 10, 12]] > 0).all()
    assert (ctas[:, 0] > 0).all() and (ctas[:, 1] > ctas[:, 0]).all()

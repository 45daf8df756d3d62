"""The chain of segment states h[s + 1] += M[s] h[s] (``qla_cp_chain``) by itself, against 64 bits: one link, links that are left out,
either direction, several sequences, and more links than the kernel looks at in one batch."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("segments, skip, reverse", [
    ([2], [], False),
    ([5, 1, 3], [], False),
    ([5, 1, 3], [1], True),
    ([38], [0, 7, 8, 20], False),
    ([300], [255, 256], False),   # the kernel takes 256 flags at a time
    ([300], [40, 43], True),
])
def test_chain(segments, skip, reverse):
    from flashqla_b200 import _cabi
    Hv, n = 2, sum(segments)
    gen = torch.Generator(device="cuda").manual_seed(n)
    h = torch.randn(n, Hv, 128, 128, generator=gen, device="cuda")
    M = torch.randn(n, Hv, 128, 128, generator=gen, device="cuda") * (0.9 / 128 ** 0.5)
    limit = torch.ones(n, Hv, dtype=torch.int32, device="cuda")
    limit[skip, 0] = 0  # (of one head only)
    first = torch.tensor([0] + segments).cumsum(0).int().cuda()
    ref = h.double()
    for a, b in zip(first.tolist()[:-1], first.tolist()[1:]):
        order = list(range(a, b))
        order = order[::-1] if reverse else order
        for s, t in zip(order[:-1], order[1:]):
            for hd in range(Hv):
                if limit[s, hd]:
                    ref[t, hd] += M[s, hd].double() @ ref[s, hd]
    args = _cabi.QlaCpChainArgs(num_raw_seqs=len(segments), num_v_heads=Hv, h0=h.data_ptr(), M=M.data_ptr(),
                                m_limit=limit.data_ptr(), raw_first_seg=first.data_ptr(), reverse=int(reverse))
    _cabi.check(_cabi.lib().qla_cp_chain(args, _cabi.current_stream(h.device)), "qla_cp_chain")
    # a product loses up to 2^-21 of itself to the splitting, sums of 128 in fp32; |M| |h| is up to ten times |M h| here
    assert float((h.double() - ref).norm() / ref.norm()) <= 1e-5


def chain(h, M):
    """``h`` after the links of one sequence, by the kernel."""
    from flashqla_b200 import _cabi
    n, Hv = h.shape[:2]
    out, limit = h.clone(), torch.ones(n, Hv, dtype=torch.int32, device="cuda")
    first = torch.tensor([0, n], dtype=torch.int32, device="cuda")
    args = _cabi.QlaCpChainArgs(num_raw_seqs=1, num_v_heads=Hv, h0=out.data_ptr(), M=M.data_ptr(), m_limit=limit.data_ptr(),
                                raw_first_seg=first.data_ptr(), reverse=0)
    _cabi.check(_cabi.lib().qla_cp_chain(args, _cabi.current_stream(h.device)), "qla_cp_chain")
    return out


def test_callers_hand_the_chain_their_status_word(monkeypatch):
    """The Python callers of the chain (the native one sets it in segment_chain): the device's status word goes with every launch."""
    from flashqla_b200 import _cabi, chunk, cp, seq_parallel, utils
    seen = []

    class Recorder:
        def __getattr__(self, name):
            f = getattr(real, name)
            return f if name != "qla_cp_chain" else lambda a, stream: (seen.append((a.has_status, a.status)), f(a, stream))[1]

    real = _cabi.lib()
    monkeypatch.setattr(_cabi, "lib", Recorder)
    T, Hv = 4096, 2
    gen = torch.Generator(device="cuda").manual_seed(3)
    q, k, v = (torch.nn.functional.normalize(torch.randn(1, T, Hv, 128, generator=gen, device="cuda"), dim=-1).bfloat16() for _ in range(3))
    g, beta = -0.1 * torch.rand(1, T, Hv, generator=gen, device="cuda"), torch.rand(1, T, Hv, generator=gen, device="cuda")
    ctx = seq_parallel.slice_summary(q, k, v, g, beta)
    assert len(seen) == 2
    plan = cp.get_plan([T], Hv, q.device)
    assert plan.use_cp
    cp.segment_initial_states(plan, k, v, beta, ctx.tensors[4], ctx.tensors[5], ctx.tensors[6], None, ctx.scale, chunk._launch_fwd)
    assert seen == [(1, utils.device_status(q.device).data_ptr())] * 3
    utils.check_device_status()


def plain(h, M):
    """The same in the type of ``h``, sums of 128 products one after the other."""
    out = h.clone()
    for s in range(len(h) - 1):
        acc = torch.zeros_like(out[0])
        for j in range(128):
            acc += M[s][:, :, j, None] * out[s][:, None, j]
        out[s + 1] += acc
    return out


@pytest.mark.parametrize("segments, norm", [(2, 0.9), (38, 0.9), (38, 1.0)])
def test_chain_is_as_exact_as_fp32(segments, norm):
    gen = torch.Generator(device="cuda").manual_seed(segments)
    h = torch.randn(segments, 2, 128, 128, generator=gen, device="cuda")
    M = torch.randn(segments, 2, 128, 128, generator=gen, device="cuda") * (norm / 128 ** 0.5)
    ref = plain(h.double(), M.double())
    error = lambda x: float((x.double() - ref).norm() / ref.norm())
    assert error(chain(h, M)) <= error(plain(h, M))  # (16 terms one after the other, then a tree: 16 + 3 roundings instead of 128)


def test_chain_beyond_the_range_of_a_splitting():
    """Values up to the end of the fp32 range, and infinities that stay in their column."""
    gen = torch.Generator(device="cuda").manual_seed(1)
    h = 1e37 * torch.randn(3, 1, 128, 128, generator=gen, device="cuda")
    M = torch.randn(3, 1, 128, 128, generator=gen, device="cuda") * (0.5 / 128 ** 0.5)
    h[0, 0, 5, 7] = float("inf")
    out, ref = chain(h, M), plain(h, M)
    assert torch.equal(torch.isfinite(out), torch.isfinite(ref)) and torch.equal(torch.isnan(out), torch.isnan(ref))
    fine = torch.isfinite(ref)
    assert float((out[fine].double() - ref[fine].double()).norm() / ref[fine].double().norm()) <= 1e-5

"""The preparation kernel's own outputs, ``A`` and ``w``, against a triangular solve in 64 bits, where its work items can go wrong:
sequences that end inside the first or second chunk of a pair (also many in a row), v-head groups that are spread over several
items, and the in-kernel norm."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def solve(k, g, beta):
    """``A [T, Hv, 64]`` and ``w [T, Hv, 128]`` of one sequence in 64 bits."""
    T, Hk, Hv = k.shape[0], k.shape[1], g.shape[1]
    A = torch.zeros(T, Hv, 64, dtype=torch.float64, device=k.device)
    w = torch.zeros(T, Hv, 128, dtype=torch.float64, device=k.device)
    for t0 in range(0, T, 64):
        kk = k[t0:t0 + 64].repeat_interleave(Hv // Hk, 1).permute(1, 0, 2)
        gc, b = g[t0:t0 + 64].cumsum(0).t(), beta[t0:t0 + 64].t()
        n = kk.shape[1]
        decay = torch.exp((gc[:, :, None] - gc[:, None, :]).tril())
        L = (b[:, :, None] * decay * (kk @ kk.transpose(1, 2))).tril(-1)
        eye = torch.eye(n, dtype=torch.float64, device=k.device)
        X = torch.linalg.solve_triangular(eye + L, eye.expand(Hv, n, n), upper=False, unitriangular=True)
        A[t0:t0 + n, :, :n] = X.permute(1, 0, 2)
        w[t0:t0 + n] = -(X @ ((b * torch.exp(gc))[:, :, None] * kk)).permute(1, 0, 2)
    return A, w


@pytest.mark.parametrize("lens, heads, norm", [
    ([1, 64, 65, 127, 128, 129, 63, 200], (2, 4), False),
    ([40] * 700 + [300], (2, 2), False),        # several items per CTA, none of them with a second chunk
    ([130, 3] * 300, (2, 4), True),
    ([64 * 17 + 5], (1, 6), False),             # a small grid: the six v-heads as items of their own
    ([777], (4, 8), True),
])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_a_and_w(lens, heads, norm, dtype):
    import flashqla_b200 as fq
    gen = torch.Generator(device="cuda").manual_seed(len(lens))
    T, (Hk, Hv) = sum(lens), heads
    q, k, v = (torch.randn(1, T, n, 128, generator=gen, device="cuda") for n in (Hk, Hk, Hv))
    if not norm:
        k = torch.nn.functional.normalize(k, dim=-1)
    q, k, v = q.to(dtype), k.to(dtype), v.to(dtype)
    g = torch.nn.functional.logsigmoid(torch.randn(1, T, Hv, generator=gen, device="cuda")) / 4
    beta = torch.sigmoid(torch.randn(1, T, Hv, generator=gen, device="cuda"))
    cu = torch.tensor([0] + lens).cumsum(0).int().cuda()
    out = fq.chunk_gated_delta_rule_fwd(q, k, v, g, beta, cu_seqlens=cu, use_qk_l2norm_in_kernel=norm, output_w=True)
    fq.check_device_status()
    kd = k[0].double()
    if norm:
        kd = kd * torch.rsqrt(kd.pow(2).sum(-1, keepdim=True) + 1e-6)
    eps = torch.finfo(dtype).eps / 2  # largest relative error of one rounding to the 16-bit type
    for i in range(0, len(lens), max(1, len(lens) // 40)):
        a, b = int(cu[i]), int(cu[i + 1])
        A, w = solve(kd[a:b], g[0, a:b].double(), beta[0, a:b].double())
        # A is rounded once, its lower left 32 x 32 blocks come from TF32 factors (2^-11 each, three of them)
        assert float((out[1][0, a:b].double() - A).abs().max()) <= float(A.abs().max()) * (eps + 3 * 2.0 ** -11)
        # w: A diag(beta gamma) rounded, the product rounded, and A's own error
        assert float((out[5][0, a:b].double() - w).norm() / w.norm()) <= 3 * eps + 3 * 2.0 ** -11


def test_off_diagonal_blocks_are_as_exact_as_fp32():
    """The 16 x 16 blocks beside the diagonal inside the two 32 x 32 diagonal blocks, where the inverse grows (alike keys, no decay): the
    share of fp16 entries that are not the exact value's nearest.  Forward substitution in fp32 gives 4.8 % (of rounding K K^T and the
    products), factors of 21 bits 7.5 %."""
    import flashqla_b200 as fq
    gen = torch.Generator(device="cuda").manual_seed(0)
    T, Hk, Hv = 4096, 4, 8
    k = 0.3 * torch.randn(T, Hk, 128, generator=gen, device="cuda") + torch.randn(1, Hk, 128, generator=gen, device="cuda")
    k = torch.nn.functional.normalize(k, dim=-1).half()
    q, v = (torch.randn(1, T, n, 128, generator=gen, device="cuda").half() for n in (Hk, Hv))
    g, beta = torch.zeros(T, Hv, device="cuda"), 0.5 + 0.5 * torch.rand(T, Hv, generator=gen, device="cuda")
    out = fq.chunk_gated_delta_rule_fwd(q, k[None], v, g[None], beta[None])
    fq.check_device_status()
    A, ref = out[1][0].view(-1, 64, Hv, 64), solve(k.double(), g.double(), beta.double())[0].half().view(-1, 64, Hv, 64)
    wrong = [(A[:, d + 16:d + 32, :, d:d + 16] != ref[:, d + 16:d + 32, :, d:d + 16]).double().mean() for d in (0, 32)]
    assert float(sum(wrong)) / 2 <= 0.06


@pytest.mark.parametrize("dtype", [torch.bfloat16])
def test_values_up_to_the_end_of_the_range(dtype):
    """Gates that grow: entries of A up to 1e36 (a splitting by 8193 x would overflow from 4e34 on)."""
    import flashqla_b200 as fq
    gen = torch.Generator(device="cuda").manual_seed(2)
    T, H = 64, 2
    k = torch.nn.functional.normalize(torch.randn(T, H, 128, generator=gen, device="cuda"), dim=-1).to(dtype)
    g, beta = torch.full((T, H), 1.39, device="cuda"), torch.rand(T, H, generator=gen, device="cuda")
    v = torch.randn(1, T, H, 128, generator=gen, device="cuda").to(dtype)
    A = fq.chunk_gated_delta_rule_fwd(v, k[None], v, g[None], beta[None])[1][0]
    fq.check_device_status()
    ref = solve(k.double(), g.double(), beta.double())[0]
    assert float(ref.abs().max()) > 1e35
    # relative to what the decay makes of an entry: one rounding to 16 bits, three TF32 factors
    gc = g.double().cumsum(0)
    scale = torch.exp(gc[:, None, :] - gc[None, :, :]).transpose(1, 2)
    assert float(((A.double() - ref) / scale).abs().max()) <= float((ref / scale).abs().max()) * (torch.finfo(dtype).eps / 2 + 3 * 2.0 ** -11)

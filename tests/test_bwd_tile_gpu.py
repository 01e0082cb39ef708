"""The whole TF32 backward of sequences of one tile (128 rows) in one kernel: its forms, at the edges of its 16-column blocks and of the tile."""
import pytest

import helpers as hp
from helpers import pkg, to_dev

pytestmark = pytest.mark.gpu


# B x H: a CTA for either side of a head, one for both (from 75 heads on a 148-SM device), two and three waves (of causal heads), and past the
# last wave that the rule takes
@pytest.mark.parametrize("B,H", [(1, 3), (2, 37), (1, 75), (5, 30), (4, 111), (5, 89)])
@pytest.mark.parametrize("S", [1, 15, 16, 17, 33, 64, 100, 127, 128])
@pytest.mark.parametrize("causal", [True, False])
def test_one_tile_backward_against_float64(B, H, S, causal):
    import torch
    from test_split_gpu import _reference
    p = pkg()
    from oracle.attn_oracle import Oracle
    orc = Oracle()
    q, k, v, go = to_dev(*(orc.fill_normal((B, S, H * 64), 700 + S, i) for i in range(4)))
    scale = hp.default_scale(64)
    out, lse = p.forward(q, k, v, H, scale, causal)

    def run(f, o, **kw):
        delta = torch.full((B, H, S), 9.0, device="cuda")
        got = f(q, k, v, o, go, lse, H, scale, causal, delta_buf=delta, **kw)[:3]
        assert p.sync_status() == 0
        return tuple(got) + (delta,)

    got, again = run(p.backward, out), run(p.backward, out)
    two = run(p.backward_profile, out)  # timed kernel by kernel, so always in two
    o = out.clone()
    in_place = run(p.backward, o, d_q=o)  # d_q in the place of O, which only dQ's side reads
    refs = _reference(torch, q, k, v, go, H, scale, causal, 0)[2:]
    for n, name in enumerate(("dq", "dk", "dv")):
        assert torch.equal(got[n], again[n]) and torch.equal(got[n], in_place[n]), name  # no atomics: the same bits every time
        size = max(1.0, float(refs[n].abs().max()))
        err, err_two = (float((x[n].double() - refs[n]).abs().max()) for x in (got, two))
        assert err <= hp.TOL_GRAD_REL_TF32 * size, name
        # operands rounded to 11 bits either way, P on the dK side too: half a unit of that is all that may lie between the two
        assert err <= err_two + 2.0 ** -12 * size, name
    assert torch.equal(got[3], two[3])  # the row sums are the same sums


@pytest.mark.parametrize("S,D,bf16", [(100, 64, False), (300, 64, False), (300, 64, True), (300, 128, True)])
@pytest.mark.parametrize("scale", [1e-30, 1e-35, 3e-37, 5e-38, 2e-38, 1e-40])
def test_backward_with_a_scale_that_makes_scores_equal(S, D, bf16, scale):
    """The logsumexp enters the score products divided by the scale. Such a scale leaves uniform probabilities, dV = means, and dQ = dK = 0 but for the scale."""
    import torch
    p = pkg()
    from oracle.attn_oracle import Oracle
    orc = Oracle()
    H = 3
    q, k, v, go = to_dev(*(orc.fill_normal((1, S, H * D), 500 + S, i) for i in range(4)))
    fwd, bwd = (p.forward_bf16, p.backward_bf16) if bf16 else (p.forward, p.backward)
    if bf16:
        q, k, v, go = (x.to(torch.bfloat16) for x in (q, k, v, go))
    prev = p.set_variant(p.VARIANT_TENSOR)
    try:
        out, lse = fwd(q, k, v, H, scale, True)
        d_q, d_k, d_v = bwd(q, k, v, out, go, lse, H, scale, True)[:3]
        assert p.sync_status() == 0
    finally:
        p.set_variant(prev)
    weights = 1.0 / torch.arange(1, S + 1, device="cuda", dtype=torch.float64)
    ref = torch.flip(torch.cumsum(torch.flip(go.double() * weights[None, :, None], [1]), 1), [1])
    tol = 2.0 ** -7 if bf16 else hp.TOL_GRAD_REL_TF32
    assert float((d_v.double() - ref).abs().max()) <= tol * max(1.0, float(ref.abs().max()))
    for d in (d_q, d_k):
        assert float(d.double().abs().max()) <= 1e4 * scale


def test_large_logsumexps_leave_no_bias():
    """The logsumexp is subtracted from scores that are about as large (here |lse| is 290). Operands of eight bits, so that products are exact: what is left
    are errors of either sign, P's rounding to 2^-12 and the logsumexp's own to 290 * 2^-24 = 1.7e-5 of P, over 24000 rows and 1.5 M elements 3e-7 in
    the mean, and what the accumulators cut off the scores. Sums that began with lse / scale would lose 6e-6 in the mean."""
    import torch
    from test_split_gpu import _reference
    p = pkg()
    B, H, S, D = 2, 12, 1000, 64
    for seed in (1, 2):
        torch.manual_seed(seed)
        q, k, v, go = (torch.randn(B, S, H * D, device="cuda").to(torch.bfloat16).float() * f for f in (64.0, 1.0, 1.0, 1.0))
        _, lse, _, _, ref = _reference(torch, q, k, v, go, H, D ** -0.5, True, 0)
        out, _ = p.forward(q, k, v, H, D ** -0.5, True)
        got = p.backward_block(q, k, v, go, lse.float(), p.delta(out, go, H), H, D ** -0.5, True)[2]
        assert p.sync_status() == 0
        assert abs(float(((got.double() - ref) * ref).sum() / (ref * ref).sum())) <= 2e-6


@pytest.mark.parametrize("D,bf16", [(64, False), (64, True), (128, True)])
def test_an_infinite_row_sum_stays_infinite(D, bf16):
    """delta = inf of one query: its dS is -inf at every key that it sees, and so is dK, with the sign of its Q (or NaN at Q = 0)."""
    import torch
    p = pkg()
    S, H, row = 200, 2, 77
    torch.manual_seed(3)
    q, k, v, go = (torch.randn(1, S, H * D, device="cuda") for _ in range(4))
    q = torch.where(q == 0, 1.0, q)
    f = (lambda x: x.to(torch.bfloat16)) if bf16 else (lambda x: x)
    q, k, v, go = map(f, (q, k, v, go))
    out, lse = (p.forward_bf16 if bf16 else p.forward)(q, k, v, H, D ** -0.5, False)
    delta = (p.delta_bf16 if bf16 else p.delta)(out, go, H)
    delta[0, 1, row] = float("inf")
    d_k, d_v = (p.backward_block_bf16 if bf16 else p.backward_block)(q, k, v, go, lse, delta, H, D ** -0.5, False)[1:3]
    assert p.sync_status() == 0
    assert torch.isfinite(d_v).all() and torch.isfinite(d_k[..., :D]).all()
    assert torch.equal(d_k[0, :, D:].float(), (-torch.sign(q[0, row, D:].float()) * float("inf")).expand(S, D))

"""fp32 attention on the tensor cores with operands cut into three bf16 parts (head sizes other than 64, four steps of 64 keys or more): the forms
that its rules choose between, at the edges of its tiles, against float64. Two bars: 2e-5 of the result's scale for its largest error, as for the other
fp32 kernels, and 1.5e-6 for the relative 2-norm error, of which the kernels take 1e-7 to 3.1e-7. A product that lost one of its three parts would be 1e-5
off in the 2-norm; its largest error alone could pass."""
import os
import shutil
import subprocess
import sys
import textwrap

import pytest

import helpers as hp
from helpers import pkg, to_dev

pytestmark = pytest.mark.gpu


def _reference(torch, q, k, v, go, H, scale, causal, shift):
    q4, k4, v4, g4 = (t.double().view(t.shape[0], t.shape[1], H, -1).transpose(1, 2) for t in (q, k, v, go))
    s = q4 @ k4.transpose(2, 3) * scale
    if causal:
        hidden = torch.arange(k.shape[1], device="cuda")[None, :] > torch.arange(q.shape[1], device="cuda")[:, None] + shift
        s = s.masked_fill(hidden, -torch.inf)
    lse = torch.logsumexp(s, -1)
    pr = torch.exp(s - torch.where(torch.isinf(lse), 0.0, lse)[..., None])
    o = pr @ v4
    ds = pr * (g4 @ v4.transpose(2, 3) - (g4 * o).sum(-1, keepdim=True))
    back = lambda t: t.transpose(1, 2).reshape(t.shape[0], t.shape[2], -1)
    return back(o), lse, back(ds @ k4 * scale), back(ds.transpose(2, 3) @ q4 * scale), back(pr.transpose(2, 3) @ g4)


# B x H: one CTA a block, two (few blocks), four (very few, and eight steps). Sequences: just over four steps, whole tiles, a row more, keys ahead of
# the queries, queries that see no key, all keys visible.
@pytest.mark.parametrize("B,H,Sq,Sk,causal,shift", [
    (8, 20, 193, 193, True, 0), (8, 20, 257, 257, True, 0), (4, 20, 130, 320, False, 0),
    (2, 3, 193, 193, True, 0), (2, 3, 256, 256, True, 0), (2, 3, 100, 321, True, 221), (2, 3, 300, 420, True, -100), (2, 3, 321, 100, True, -150),
    (1, 1, 449, 449, True, 0), (1, 2, 640, 640, False, 0)])
@pytest.mark.parametrize("D", [4, 32, 36, 80, 96, 100, 128])
def test_split_against_float64(B, H, Sq, Sk, causal, shift, D):
    import torch
    p = pkg()
    from oracle.attn_oracle import Oracle
    orc = Oracle()
    q, go = (orc.fill_normal((B, Sq, H * D), 900 + Sq + D, i) for i in (0, 3))
    k, v = (orc.fill_normal((B, Sk, H * D), 900 + Sq + D, i) for i in (1, 2))
    q, k, v, go = to_dev(q, k, v, go)
    scale = hp.default_scale(D)

    def run():
        out, lse = p.forward(q, k, v, H, scale, causal, causal_shift=shift)
        delta = p.delta(out, go, H)
        got = (out, lse) + tuple(p.backward_block(q, k, v, go, lse, delta, H, scale, causal, causal_shift=shift))
        assert p.sync_status() == 0
        return got

    got, again = run(), run()
    for got_t, again_t, ref, name in zip(got, again, _reference(torch, q, k, v, go, H, scale, causal, shift), ("out", "lse", "dq", "dk", "dv")):
        assert torch.equal(got_t, again_t), name  # no atomics: the same bits every time
        seen = torch.isfinite(ref)
        assert torch.equal(torch.isfinite(got_t), seen), name
        ref = torch.where(seen, ref, 0.0)
        err = torch.where(seen, got_t, 0.0).double() - ref
        assert float(err.abs().max()) <= (1e-6 if name == "lse" else 2e-5) * max(1.0, float(ref.abs().max())), name
        assert float(err.norm()) <= 1.5e-6 * float(ref.norm()), name
    prev = p.set_variant(p.VARIANT_SIMT)
    try:
        other = run()
    finally:
        p.set_variant(prev)
    assert not torch.equal(got[4], other[4])  # dV: the rule did choose another kernel


@pytest.mark.parametrize("B,H,S,D", [(1, 1, 600, 96), (1, 4, 333, 32), (4, 12, 260, 128)])
def test_split_on_another_stream_and_in_place(B, H, S, D):
    """Inputs that another stream is still writing when the calls are made there; the output in the place of Q, and dQ in the place of the output."""
    import torch
    p = pkg()
    torch.manual_seed(D)
    x = [torch.randn(B, S, H * D, device="cuda") for _ in range(4)]
    scale = hp.default_scale(D)
    out, lse = p.forward(*x[:3], H, scale, True)
    want = [out, lse] + list(p.backward(*x[:3], out, x[3], lse, H, scale, True)[:3])
    torch.cuda.synchronize()
    side = torch.cuda.Stream()
    late = [torch.full_like(t, float("nan")) for t in x]
    busy = torch.randn(4096, 4096, device="cuda")
    torch.cuda.synchronize()
    with torch.cuda.stream(side):
        for _ in range(20):
            busy = busy @ busy * 1e-3  # some milliseconds ahead of the inputs
        for a, b in zip(late, x):
            a.copy_(b)
        place = late[0].clone()
        got_lse = p.forward(place, late[1], late[2], H, scale, True, out=place)[1]
        got_out = place.clone()
        got = p.backward(*late[:3], place, late[3], got_lse, H, scale, True, d_q=place)[:3]
    side.synchronize()
    assert p.sync_status() == 0
    for name, a, b in zip(("out", "lse", "dq", "dk", "dv"), (got_out, got_lse, *got), want):
        assert torch.equal(a, b), name


# operands: normal; just above 1 + 2^-8 and 1 + 2^-7 in size, where the second and third of three bf16 parts are largest; scores of +-30 and more
@pytest.mark.parametrize("operands", ["normal", "1+2^-8", "1+2^-7", "large scores"])
@pytest.mark.parametrize("B,H,S,D,causal", [(2, 6, 400, 32, True), (1, 8, 333, 80, True), (2, 8, 1000, 128, True), (1, 4, 260, 112, False), (1, 4, 1300, 48, True)])
def test_split_is_as_exact_as_fp32_arithmetic(B, H, S, D, causal, operands):
    """Error against float64 (2-norm, relative), next to that of the kernel that computes in fp32 throughout: no larger in O and the gradients. The
    logsumexp bears the rounding of scale * log2 e (2^-24 of the scores at most) and its own (2^-24 of itself): 2^-23."""
    import torch
    p = pkg()
    torch.manual_seed(S + D)
    x = [torch.randn(B, S, H * D, device="cuda") for _ in range(4)]
    if operands.startswith("1+"):
        x = [torch.sign(t) * (1 + 2.0 ** -int(operands[-1]) + 2.0 ** -23 * torch.randint(-99, 100, t.shape, device="cuda")) for t in x]
    elif operands == "large scores":
        x[0] *= 10
    q, k, v, go = x
    scale = hp.default_scale(D)
    ref = _reference(torch, q, k, v, go, H, scale, causal, 0)
    errors = []
    for variant in (p.VARIANT_AUTO, p.VARIANT_SIMT):
        prev = p.set_variant(variant)
        try:
            out, lse = p.forward(q, k, v, H, scale, causal)
            got = (out, lse) + tuple(p.backward(q, k, v, out, go, lse, H, scale, causal)[:3])
            assert p.sync_status() == 0
        finally:
            p.set_variant(prev)
        errors.append([float((g.double() - r).norm() / r.norm()) for g, r in zip(got, ref)])
    for name, a, b in zip(("out", "lse", "dq", "dk", "dv"), *errors):
        assert a <= (2.0 ** -23 if name == "lse" else b), (name, a, b)


def _visible_only(torch, q, k, v, go, lse, delta, scale, causal):
    """One head in float64, products summed over the visible pairs alone (0 * inf of a hidden pair is no term): out, dq, dk, dv of [S, D]."""
    S = q.shape[0]
    hidden = torch.arange(S, device="cuda")[None, :] > torch.arange(S, device="cuda")[:, None] if causal else torch.zeros((S, S), dtype=torch.bool, device="cuda")
    q, k, v, go, lse, delta = (t.double() for t in (q, k, v, go, lse, delta))
    each = lambda w, x, dim: torch.where(hidden[..., None], 0.0, w[..., None] * x.unsqueeze(1 - dim)).sum(dim)  # over queries (0) or keys (1)
    s = (q[:, None] * k[None]).sum(-1) * scale
    top = torch.nan_to_num(torch.where(hidden, -torch.inf, s), nan=-torch.inf, posinf=torch.inf, neginf=-torch.inf).amax(1, keepdim=True)
    w = torch.where(hidden, 0.0, torch.exp(s - torch.where(top == -torch.inf, 0.0, top)))
    out = each(w, v, 1) / w.sum(1, keepdim=True)
    pr = torch.where(hidden, 0.0, torch.exp(s - torch.where(lse == -torch.inf, torch.inf, lse)[:, None]))
    ds = torch.where(hidden, 0.0, pr * ((go[:, None] * v[None]).sum(-1) - delta[:, None]))
    return out, each(ds, k, 1) * scale, each(ds, q, 0) * scale, each(pr, go, 0)


# where: tensor, row, value. A CTA a block, two, four.
@pytest.mark.parametrize("tensor,value", [("v", float("inf")), ("v", float("nan")), ("v", 3.4e38), ("k", float("-inf")), ("k", float("nan")), ("q", float("inf")),
                                          ("go", float("-inf"))])
@pytest.mark.parametrize("H,S,D,causal", [(60, 260, 128, True), (2, 300, 32, True), (1, 600, 96, True), (2, 449, 36, False)])
def test_split_with_operands_that_are_not_finite(H, S, D, causal, tensor, value):
    """What fp32 arithmetic gives: an infinite V an infinite O, a score of -inf a probability of zero; rows that do not see it stay as they are."""
    import torch
    p = pkg()
    torch.manual_seed(S)
    x = {n: torch.randn(1, S, H * D, device="cuda") for n in ("q", "k", "v", "go")}
    x["q"][..., ::D] = x["q"][..., ::D].abs() + 0.1  # against an infinite K in the head's first dim
    scale = hp.default_scale(D)

    def run():
        out, lse = p.forward(x["q"], x["k"], x["v"], H, scale, causal)
        delta = p.delta(out, x["go"], H)
        got = (out,) + tuple(p.backward_block(x["q"], x["k"], x["v"], x["go"], lse, delta, H, scale, causal)[:3])
        assert p.sync_status() == 0
        return lse, delta, got

    clean = run()[2]
    row, head = S // 2 + 9, H - 1
    x[tensor][0, row, head * D] = value
    lse, delta, got = run()
    cut = slice(head * D, (head + 1) * D)
    ref = _visible_only(torch, *(x[n][0, :, cut] for n in ("q", "k", "v", "go")), lse[0, head], delta[0, head], scale, causal)
    for name, a, c, r in zip(("out", "dq", "dk", "dv"), got, clean, ref):
        if value == 3.4e38 and name in ("dq", "dk"):  # dP is past fp32
            continue
        assert torch.equal(a[..., :head * D], c[..., :head * D]), name
        a, r = a[0, :, cut], r.float()
        assert torch.equal(torch.isnan(a), torch.isnan(r)), name
        assert torch.equal(torch.isinf(a) * torch.sign(a).nan_to_num(), torch.isinf(r) * torch.sign(r).nan_to_num()), name
        seen = torch.isfinite(r)
        a, r = torch.where(seen, a, 0.0).double(), torch.where(seen, r, 0.0).double()
        assert bool(((a - r).abs() <= 2e-5 * torch.clamp(r.abs(), min=1.0)).all()), name
    if causal:  # rows that do not see it
        before = row if tensor in ("k", "v") else 0
        assert torch.isfinite(got[0][:, :before]).all() and torch.isfinite(got[1][:, :before]).all()
        if tensor in ("q", "go"):
            assert torch.isfinite(got[2][:, row + 1:]).all() and torch.isfinite(got[3][:, row + 1:]).all()


ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
OTHER_REGISTERS = textwrap.dedent("""
    import sys
    sys.path.insert(0, {root!r})
    import torch
    from __graft_entry__ import load_package
    p = load_package()
    p.LIB_PATH = {lib!r}
    torch.manual_seed(1)
    for B, H, S, D in ((1, 2, 449, 36), (2, 3, 300, 96), (4, 15, 260, 128)):
        q, k, v, go = (torch.randn(B, S, H * D, device="cuda") for _ in range(4))
        got = []
        for variant in (p.VARIANT_AUTO, p.VARIANT_SIMT):
            p.set_variant(variant)
            out, lse = p.forward(q, k, v, H, D ** -0.5, True)
            got.append([out, lse] + list(p.backward(q, k, v, out, go, lse, H, D ** -0.5, True)[:3]))
            assert p.sync_status() == 0
        assert all(torch.equal(a, b) for a, b in zip(*got))
    print("SAME")
""")


def test_split_kernels_with_other_registers_leave_calls_to_the_simt_kernels(tmp_path):
    """A library whose split kernels are taken to have been built with 127 registers a thread launches none of them, and answers all the same."""
    if shutil.which("nvcc") is None and not os.path.exists("/usr/local/cuda/bin/nvcc"):
        pytest.skip("nvcc is not available: the variant cannot be built here")
    out_dir = str(tmp_path / "lib")
    lib = os.path.join(out_dir, "libdarkforest_kernels.so")
    r = subprocess.run(["make", "-C", os.path.join(ROOT, "dark-forest_b200"), "-j8", f"OUT={out_dir}", "EXTRA=-DDF_SPLIT_BUILT_REGS=127", lib],
                       capture_output=True, text=True, timeout=900)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-2000:]
    child = subprocess.run([sys.executable, "-c", OTHER_REGISTERS.format(root=ROOT, lib=lib)], capture_output=True, text=True, timeout=600)
    assert child.returncode == 0 and "SAME" in child.stdout, child.stdout[-3000:] + child.stderr[-3000:]

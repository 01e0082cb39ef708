"""The TF32 forward of sequences of one tile (128 rows and keys): edges of its 32-key blocks and of the tile, more keys than queries, rows that see no key."""
import pytest

import helpers as hp
from helpers import pkg, to_dev

pytestmark = pytest.mark.gpu


# B x H: few heads, two waves of two CTAs an SM, and (all keys visible) past the heads that the rule takes
@pytest.mark.parametrize("B,H", [(1, 3), (3, 111), (5, 89)])
@pytest.mark.parametrize("Sq,Sk,causal,shift", [(1, 1, True, 0), (31, 31, True, 0), (33, 33, False, 0), (64, 64, True, 0), (65, 65, False, 0), (127, 127, True, 0),
                                                (128, 128, True, 0), (128, 128, False, 0), (1, 128, True, 127), (7, 100, True, 93), (128, 40, False, 0),
                                                (100, 128, True, -50), (60, 30, True, -70)])
def test_one_tile_forward_against_float64(B, H, Sq, Sk, causal, shift):
    import torch
    from test_split_gpu import _reference
    p = pkg()
    from oracle.attn_oracle import Oracle
    orc = Oracle()
    q = orc.fill_normal((B, Sq, H * 64), 600 + Sq, 0)
    k, v = (orc.fill_normal((B, Sk, H * 64), 600 + Sq, i) for i in (1, 2))
    q, k, v = to_dev(q, k, v)
    scale = hp.default_scale(64)
    ref_o, ref_lse = _reference(torch, q, k, v, torch.zeros_like(q), H, scale, causal, shift)[:2]
    seen = torch.isfinite(ref_lse)
    buf = torch.empty(B * Sq * H * 64 + 4, device="cuda")
    first = None
    for out in (None, buf[4:].view(B, Sq, H * 64)):  # the second: 16-byte stores
        o, lse = p.forward(q, k, v, H, scale, causal, causal_shift=shift, out=out)
        assert p.sync_status() == 0
        first = o if first is None else first
        assert torch.equal(o, first)
        assert torch.equal(torch.isfinite(lse), seen)
        assert float((o.double() - ref_o.nan_to_num(0.0)).abs().max()) <= hp.TOL_O_TF32
        if seen.any():
            assert float((lse[seen].double() - ref_lse[seen]).abs().max()) <= hp.TOL_LSE_TF32

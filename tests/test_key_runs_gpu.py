"""The K kernel for up to 64 query blocks per kv head (D = 64: 128): its blocks walk runs of key tiles, two blocks per SM, a run going on into the next head.  Numbers of
tiles around the blocks that are resident, query blocks around the 32 and 64 columns of an accumulator and the halves of them that a warp writes, ragged
last tiles, tokens split over buffers: codes, scales, means and delta_s as the oracle forms them and as a call on one head alone gives them."""
import pytest
import torch

from oracle import sage3_oracle as O
from sageattention_b200 import Sage3Problem

pytestmark = pytest.mark.gpu


def _workspace(p, B, Hkv):
    """What the K kernel writes, per kv head."""
    ws, lay = p.ws.buf, p.ws.layout
    d = p.desc
    nk_p = (d.Nk + 127) // 128 * 128
    def at(off, n):
        return ws[off: off + n].clone()
    km = at(lay.km, B * Hkv * d.D * 2).view(B * Hkv, -1)
    codes = at(lay.k_codes, B * Hkv * nk_p * d.D // 2).view(B * Hkv, -1)
    sf = at(lay.k_sf, B * Hkv * nk_p * d.D // 16).view(B * Hkv, -1)
    nqm = lay.nqm
    delta = at(lay.delta, B * d.Hq * nqm * nk_p * 2).view(B * Hkv, -1)
    return km, codes, sf, delta


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("group,Nq,tiles,heads", [
    (1, 1, 37, 8),               # 296 tiles: one per block on 148 SMs
    (8, 1, 99, 3),               # 297: one block has two
    (3, 128 * 5 + 1, 98, 3),     # 18 query blocks, 294 tiles
    (2, 128 * 8, 37, 13),        # 16, 481 tiles: one half of an accumulator of 32 columns
    (1, 128 * 17, 37, 13),       # 17
    (1, 128 * 32, 50, 12),       # 32: all columns of it
    (1, 128 * 33, 50, 12),       # 33: an accumulator of 64 columns
    (7, 128 * 9, 45, 9),         # 63
    (4, 128 * 16, 61, 10),       # 64
    (4, 128 * 16, 33, 12),       # 64, 396 tiles: D = 64 has a block per tile
    (4, 128 * 16, 33, 15),       # 64, 495 tiles
    (5, 128 * 13, 40, 10),       # 65: D = 64 has an accumulator of 128 columns
    (8, 128 * 16, 40, 10),       # 128
    (8, 1, 100, 40),             # 4 000 tiles
])
def test_runs_of_key_tiles(cuda_device, D, group, Nq, tiles, heads):
    g = torch.Generator(device=cuda_device).manual_seed(2000 + tiles + Nq)
    Nk = tiles * 128 - 37
    k, v = (torch.randn(1, heads, Nk, D, device=cuda_device, dtype=torch.bfloat16, generator=g) for _ in range(2))
    q = torch.randn(1, heads * group, Nq, D, device=cuda_device, dtype=torch.bfloat16, generator=g)
    k += 2 * torch.randn(heads, 1, D, device=cuda_device, dtype=torch.bfloat16, generator=g)
    whole = Sage3Problem(q, k, v)
    whole.prepass()
    got = _workspace(whole, 1, heads)
    for h in sorted({0, 1, heads // 2, heads - 1}):
        one = Sage3Problem(q[:, h * group:(h + 1) * group].contiguous(), k[:, h:h + 1].contiguous(), v[:, h:h + 1].contiguous())
        one.prepass()
        for name, a, b in zip(("mean", "codes", "scales", "delta_s"), got, _workspace(one, 1, 1)):
            assert torch.equal(a[h], b[0]), (name, h)
    # delta_s against 64 bits: one rounding to bf16, and sums of D products in 32 bits that differ in order
    h, nk_p = heads - 1, (Nk + 127) // 128 * 128
    km = got[0][h].view(torch.bfloat16)
    kp = (k[0, h].float() - km.float()).to(torch.bfloat16).double()
    nqm = whole.ws.layout.nqm
    qm = whole.ws.buf[whole.ws.layout.qm: whole.ws.layout.qm + heads * group * nqm * D * 2].view(torch.bfloat16).view(heads, group * nqm, D)[h].double()
    exact = qm @ kp.T
    mine = got[3][h].view(torch.bfloat16).view(group * nqm, nk_p)
    assert (mine[:, Nk:] == 0).all()
    bound = exact.abs() * 2.0 ** -8 + (qm.abs() @ kp.abs().T) * D * 2.0 ** -24
    assert ((mine[:, :Nk].double() - exact).abs() <= bound).all()

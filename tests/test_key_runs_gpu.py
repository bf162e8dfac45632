"""The K kernel whose blocks walk runs of key tiles, two blocks per SM, a run going on into the next head (up to 64 query blocks per kv head; D = 64: 128).  Numbers of
tiles around the blocks that are resident, query blocks around the 32, 64 and 128 columns of an accumulator and the halves of them that a warp writes, ragged
last tiles, tokens split over buffers: codes, scales, means and delta_s as a call on one head alone gives them, whose tiles have a block each, and as the oracle
and 64-bit sums do."""
import ctypes as C

import pytest
import torch

from oracle import sage3_oracle as O
from sageattention_b200 import Sage3Problem, _cabi
from tests._util import canon, deatomize_sf

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


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
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
def test_runs_of_key_tiles(cuda_device, D, group, Nq, tiles, heads, dtype):
    g = torch.Generator(device=cuda_device).manual_seed(2000 + tiles + Nq)
    Nk = tiles * 128 - 37
    k, v = (torch.randn(1, heads, Nk, D, device=cuda_device, dtype=dtype, generator=g) for _ in range(2))
    q = torch.randn(1, heads * group, Nq, D, device=cuda_device, dtype=dtype, generator=g)
    k += 2 * torch.randn(heads, 1, D, device=cuda_device, dtype=dtype, generator=g)
    whole = Sage3Problem(q, k, v)
    whole.prepass()
    got = _workspace(whole, 1, heads)
    for h in sorted({0, 1, heads // 2, heads - 1}):
        one = Sage3Problem(q[:, h * group:(h + 1) * group].contiguous(), k[:, h:h + 1].contiguous(), v[:, h:h + 1].contiguous())
        one.prepass()
        for name, a, b in zip(("mean", "codes", "scales", "delta_s"), got, _workspace(one, 1, 1)):
            assert torch.equal(a[h], b[0]), (name, h)
    # the tokens of K and V in two buffers that meet inside a tile
    n, strides = (Nk + 1) // 2, (C.c_int64 * 3)
    parts = []
    cut = [[x[:, :, i * n:(i + 1) * n].contiguous() for i in range(2)] for x in (k, v)]
    cut = [[torch.nn.functional.pad(x, (0, 0, 0, n - x.shape[2])) for x in pieces] for pieces in cut]
    for pieces, rows in (([q], Nq), (cut[0], n), (cut[1], n)):
        p = _cabi.Sage3Parts()
        p.parts, p.rows_per_part = len(pieces), rows
        for i, x in enumerate(pieces):
            p.base[i] = x.data_ptr()
        parts.append(p)
    split = Sage3Problem(q, k, v)
    split.ws.buf.fill_(255)
    split.desc.k_stride = split.desc.v_stride = strides(heads * n * D, n * D, D)
    assert _cabi.lib().sage3_prepass_parts(C.byref(split.desc), *map(C.byref, parts), split.ws.buf.data_ptr(), torch.cuda.current_stream().cuda_stream) == 0
    assert split.check_status() == 0
    for name, a, b in zip(("mean", "codes", "scales", "delta_s"), got, _workspace(split, 1, heads)):
        assert torch.equal(a, b), name
    # the mean within one rounding of the exact one; codes and scales of what it leaves are the oracle's
    h, nk_p = heads - 1, (Nk + 127) // 128 * 128
    km = got[0][h].view(dtype)
    eps = torch.finfo(dtype).eps
    mean = k[0, h].double().mean(0)
    assert ((km.double() - mean).abs() <= eps * mean.abs() + 1e-6).all()
    kp = (k[0, h].float() - km.float()).to(dtype)
    codes, scales, _ = O.quant_microblocks(O.pad_rows(kp.cpu()))
    assert torch.equal(canon(O.unpack_nibbles(got[1][h].cpu().view(nk_p, D // 2))), canon(codes))
    assert torch.equal(deatomize_sf(got[2][h].cpu(), 1, nk_p // 128, D // 64)[0], scales)
    # delta_s against 64 bits: one rounding to 16, and sums of D products in 32 bits that differ in order
    kp, nqm = kp.double(), whole.ws.layout.nqm
    qm = whole.ws.buf[whole.ws.layout.qm: whole.ws.layout.qm + heads * group * nqm * D * 2].view(dtype).view(heads, group * nqm, D)[h].double()
    exact = qm @ kp.T
    mine = got[3][h].view(dtype).view(group * nqm, nk_p)
    assert (mine[:, Nk:] == 0).all()
    bound = exact.abs() * eps + (qm.abs() @ kp.abs().T) * D * 2.0 ** -24
    assert ((mine[:, :Nk].double() - exact).abs() <= bound).all()

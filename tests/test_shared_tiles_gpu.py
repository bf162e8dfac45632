"""Last rounds of the attention kernel dealt out by key blocks: a query tile's keys may then be walked by two CTAs, the second going on from the accumulator
the first leaves.  Numbers of pairs of tiles around one round and one and a half rounds of all SMs, one and two tiles per head, odd and even numbers of them, masks
aligned at the bottom right, ragged ends: the bits of calls on one head alone, whose tiles are not shared, and the oracle's result."""
import ctypes as C

import pytest
import torch

from oracle import sage3_oracle as O
from sageattention_b200 import Sage3Problem, _cabi, sageattn3

pytestmark = pytest.mark.gpu


# heads, of a kv head, queries, keys, mask; rounds of whole pairs ahead of the slots on 148 SMs (None: nothing is dealt out by blocks), which
# tests/test_split_plan.py holds against the plan
CASES = [
    (75, 1, 200, 2048, False, 0),         # 75 pairs on 148 SMs: just more than half a round
    (74, 1, 200, 2048, False, None),      # half a round: single tiles, nothing shared
    (136, 1, 256, 12000, False, 0),       # 0.92 of a round
    (160, 1, 100, 5000, False, 0),        # one tile per head, a round and twelve
    (230, 1, 90, 4000, False, 0),         # ... and more than half a round
    (149, 1, 130, 2100, False, 0),        # a round and one pair: both rounds are dealt out
    (100, 4, 384, 2500, False, 0),        # odd: every other pair is one tile
    (100, 4, 384, 3200, False, 0),
    (49, 1, 330, 2100, False, 0),         # fewer tiles than SMs, in more pairs than half of these: a slot per tile
    (37, 1, 640, 3000, False, 0),         # 111 pairs, five tiles per head
    (300, 2, 129, 2048, False, 1),        # two rounds and four
    (60, 1, 1152, 4000, False, 1),        # odd, a whole round ahead: the last tiles of all heads come first
    (24, 1, 4200, 4200, False, 2),        # ... and two
    (32, 4, 1000, 9192, True, 0),         # a chunk of a prompt: 128 pairs
    (28, 7, 900, 5000, True, 0),          # 112
    (40, 5, 1153, 8000, True, 0),         # ten tiles of a head in five pairs, 200 of them
    (56, 7, 640, 4000, True, 0),          # odd, 168 pairs, 56 of them one tile
    (90, 1, 257, 2600, True, 0),          # three tiles: the first pairs are one tile
    (170, 2, 257, 2600, True, None),      # ... of which some would be in the whole rounds
    (40, 1, 1100, 6000, True, 0),         # nine tiles: 200 pairs
    (64, 8, 1000, 6000, True, 1),         # a whole round ahead under a mask
    (56, 7, 900, 5000, True, 1),
    (48, 6, 785, 4166, True, 0),          # parts of one block, of whose keys half of the rows see none
]


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("H,group,Nq,Nk,causal,rounds", CASES)
def test_shared_tiles(cuda_device, D, H, group, Nq, Nk, causal, rounds):
    g = torch.Generator(device=cuda_device).manual_seed(2100 + H)
    q = torch.randn(1, H, Nq, D, device=cuda_device, dtype=torch.bfloat16, generator=g)
    k, v = (torch.randn(1, H // group, Nk, D, device=cuda_device, dtype=torch.bfloat16, generator=g) for _ in range(2))
    p = Sage3Problem(q, k, v, is_causal=causal, return_lse=True)
    for _ in range(2):                # (the second call finds the first one's flags and accumulators in the workspace)
        p.run()
    assert p.check_status() == 0
    p.attention()                     # ... and the attention stage on its own
    assert p.check_status() == 0
    for h in range(0, H, max(1, H // 12)):
        one, lse = sageattn3(q[:, h:h + 1], k[:, h // group:h // group + 1], v[:, h // group:h // group + 1], is_causal=causal, return_lse=True)
        assert torch.equal(p.out[:, h:h + 1], one) and torch.equal(p.lse[:, h:h + 1], lse), h
    # rows of a tile around the boundaries of slots: the whole head against 64-bit attention with the oracle's gate
    h = H // 2
    ref = O.sageattn3_oracle(q[:, h:h + 1, :].cpu(), k[:, h // group:h // group + 1].cpu(), v[:, h // group:h // group + 1].cpu(), is_causal=causal) if Nk <= 3000 else None
    if ref is not None:
        assert O.cosine(p.out[:, h:h + 1].cpu(), ref) >= 0.999 and O.rel_l1(p.out[:, h:h + 1].cpu(), ref) <= 0.01


@pytest.mark.parametrize("D", [64, 128])
def test_shared_tiles_on_two_streams_and_in_a_graph(cuda_device, D):
    """Two streams whose kernels take SMs from one another, and a captured call replayed: the results of calls one after the other."""
    g = torch.Generator(device=cuda_device).manual_seed(2200 + D)
    problems = []
    for H, Nq, Nk, causal in ((32, 1000, 6000, True), (100, 384, 3200, False)):
        q = torch.randn(1, H, Nq, D, device=cuda_device, dtype=torch.bfloat16, generator=g)
        k, v = (torch.randn(1, H // 4, Nk, D, device=cuda_device, dtype=torch.bfloat16, generator=g) for _ in range(2))
        p = Sage3Problem(q, k, v, is_causal=causal)
        problems.append((p, p.run().clone()))
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in problems]
    for p, _ in problems:
        p.out.zero_()
    torch.cuda.synchronize()
    for _ in range(20):
        for (p, _), st in zip(problems, streams):
            with torch.cuda.stream(st):
                p.run()
    torch.cuda.synchronize()
    for p, want in problems:
        assert p.check_status() == 0 and torch.equal(p.out, want)
    p, want = problems[0]
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        p.run()
        p.attention()
    p.out.zero_()
    for _ in range(3):
        graph.replay()
    torch.cuda.synchronize()
    assert p.check_status() == 0 and torch.equal(p.out, want)


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("H,group,Nq,Nk,causal", [(48, 6, 785, 4166, True), (60, 4, 1152, 4000, False)])
def test_shared_tiles_with_every_option(cuda_device, D, H, group, Nq, Nk, causal):
    """fp16, one Q mean per head, a scale per head, rows of other strides, an output split over buffers: the bits of the heads alone."""
    g = torch.Generator(device=cuda_device).manual_seed(2400 + D)
    for dtype, pbm, scales, layout in ((torch.float16, True, False, "HND"), (torch.bfloat16, False, True, "NHD")):
        q = torch.randn(1, H, Nq, D, device=cuda_device, dtype=dtype, generator=g)
        k, v = (torch.randn(1, H // group, Nk, D, device=cuda_device, dtype=dtype, generator=g) for _ in range(2))
        scale = torch.rand(H, device=cuda_device, generator=g) * 0.1 + 0.05 if scales else None
        kw = dict(is_causal=causal, per_block_mean=pbm, return_lse=True)
        qkv = (q, k, v) if layout == "HND" else tuple(x.transpose(1, 2).contiguous() for x in (q, k, v))
        out, lse = sageattn3(*qkv, tensor_layout=layout, sm_scale=scale, **kw)
        out = out if layout == "HND" else out.transpose(1, 2)
        for h in range(0, H, H // 6):
            one = sageattn3(q[:, h:h + 1], k[:, h // group:h // group + 1], v[:, h // group:h // group + 1], sm_scale=None if scale is None else float(scale[h]), **kw)
            assert torch.equal(out[:, h:h + 1], one[0]) and torch.equal(lse[:, h:h + 1], one[1]), h
    # rows 8 elements apart from one another, of q, k, v and of the output (which then has no rows of 32 bytes)
    wide = [torch.zeros(*x.shape[:3], D + 8, device=cuda_device, dtype=x.dtype) for x in (q, k, v, q)]
    for w, x in zip(wide, (q, k, v)):
        w[..., :D] = x
    p = Sage3Problem(*(w[..., :D] for w in wide[:3]), is_causal=causal, sm_scale=scale, per_block_mean=False, out=wide[3][..., :D])
    assert p.q.stride(2) == D + 8 and p.out.stride(2) == D + 8
    assert torch.equal(p.run(), out) and p.check_status() == 0 and (wide[3][..., D:] == 0).all()
    # the output's tokens in three buffers that meet inside a tile
    n = (Nq + 2) // 3
    parts, pieces = _cabi.Sage3Parts(), [torch.full((1, H, n, D), float("nan"), device=cuda_device, dtype=q.dtype) for _ in range(3)]
    parts.parts, parts.rows_per_part = 3, n
    for i, t in enumerate(pieces):
        parts.base[i] = t.data_ptr()
    p.desc.o_stride = (C.c_int64 * 3)(*pieces[0].stride()[:3])
    assert _cabi.lib().sage3_attn_fwd_parts(C.byref(p.desc), p.ws.buf.data_ptr(), C.byref(parts), None, torch.cuda.current_stream().cuda_stream) == 0
    assert p.check_status() == 0 and torch.equal(torch.cat(pieces, 2)[:, :, :Nq], out)


@pytest.mark.parametrize("D", [64, 128])
def test_a_workspace_without_room_for_shared_tiles(cuda_device, D):
    """A workspace that has room for all but the flags and accumulators is accepted, and the result is the same; one that is smaller is refused."""
    g = torch.Generator(device=cuda_device).manual_seed(2300 + D)
    q = torch.randn(2, 32, 1000, D, device=cuda_device, dtype=torch.bfloat16, generator=g)
    k, v = (torch.randn(2, 32, 6000, D, device=cuda_device, dtype=torch.bfloat16, generator=g) for _ in range(2))
    want = Sage3Problem(q, k, v, is_causal=True)
    want.run()
    assert want.desc.reserved == 0
    need = Sage3Problem(q, k, v, is_causal=True, shared_tiles=False).ws.layout.total_bytes + 256
    assert need < want.ws.layout.total_bytes
    p = Sage3Problem(q, k, v, is_causal=True, workspace=torch.full((need,), 255, dtype=torch.uint8, device=cuda_device))
    for _ in range(2):
        assert torch.equal(p.run(), want.out)
    assert p.check_status() == 0
    assert torch.equal(sageattn3(q, k, v, is_causal=True, workspace=torch.empty(need, dtype=torch.uint8, device=cuda_device)), want.out)
    with pytest.raises(ValueError, match=str(need)):
        Sage3Problem(q, k, v, is_causal=True, workspace=torch.empty(need - 1, dtype=torch.uint8, device=cuda_device))

"""Walks of few key blocks, many of them per SM: V is loaded two blocks behind K (D = 128), across units too; P slots, running maxima and
barrier phases run on from unit to unit; and the number of key blocks at which D = 64 without a mask changes kernels.  A head's result
depends on its own q, k, v alone, so every comparison is for equal bits; against the oracle the gate is the one of the whole path
(cosine >= 0.999, relative L1 <= 1 %)."""
import ctypes as C

import pytest
import torch

from oracle import sage3_oracle as O
from sageattention_b200 import Sage3Problem, _cabi, sageattn3, sageattn_varlen

pytestmark = pytest.mark.gpu


def _inputs(device, B, H, Nq, Nk, D, seed):
    q, k, v = O.make_inputs(B, H, H, Nq, Nk, D, seed=seed, dtype=torch.bfloat16, k_offset_std=1.0)
    return q.to(device), k.to(device), v.to(device)


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("Nq,Nk,causal", [(130, 1, False), (1, 128, False), (130, 129, False), (257, 300, False), (130, 650, False),
                                          (130, 130, True), (300, 300, True), (257, 100, True), (640, 640, True)])
def test_units_of_few_key_blocks(cuda_device, D, Nq, Nk, causal):
    """Some five units per SM, single tiles and pairs, of one to five key blocks (causal: the tiles of a pair with different numbers, one of them
    none, but no unit without any): the same bits as the heads alone, where each is the first unit of its SM."""
    sms = torch.cuda.get_device_properties(cuda_device).multi_processor_count
    pairs = (Nq + 255) // 256
    H = 5 * sms // pairs + 3
    q, k, v = _inputs(cuda_device, 1, H, Nq, Nk, D, seed=1300 + Nq + Nk)
    out, lse = sageattn3(q, k, v, is_causal=causal, return_lse=True)
    for h in sorted({0, 1, H // 3, H // 2, H - 2, H - 1}):
        one, one_lse = sageattn3(q[:, h:h + 1], k[:, h:h + 1], v[:, h:h + 1], is_causal=causal, return_lse=True)
        assert torch.equal(out[:, h:h + 1], one) and torch.equal(lse[:, h:h + 1], one_lse), f"head {h} of {H}"
    h = H // 2
    ref = O.sageattn3_oracle(q[:, h:h + 1].cpu(), k[:, h:h + 1].cpu(), v[:, h:h + 1].cpu(), is_causal=causal)
    assert O.cosine(out[:, h:h + 1].cpu(), ref) >= 0.999 and O.rel_l1(out[:, h:h + 1].cpu(), ref) <= 0.01


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("Nq,Nk", [(2048, 512), (1000, 100), (1300, 640)])
def test_units_without_keys(cuda_device, D, Nq, Nk):
    """Causal, more queries than keys: most units have no keys, and an SM draws three and more of them behind its full ones.  No wait gives up,
    every row is written, those without keys with zeros, and the bits are those of the heads alone."""
    sms = torch.cuda.get_device_properties(cuda_device).multi_processor_count
    H = 5 * sms // ((Nq + 255) // 256) + 3
    q, k, v = _inputs(cuda_device, 1, H, Nq, Nk, D, seed=1350 + Nq)
    prob = Sage3Problem(q, k, v, is_causal=True, return_lse=True, out=torch.full_like(q, float("nan")))
    prob.lse.fill_(float("nan"))
    out, lse = prob.run(), prob.lse
    assert prob.check_status() == 0
    blind = Nq - Nk                                # the first rows
    assert (out[:, :, :blind] == 0).all() and (lse[:, :, :blind] == float("-inf")).all() and torch.isfinite(lse[:, :, blind:]).all()
    for h in sorted({0, 1, H // 3, H // 2, H - 2, H - 1}):
        one, one_lse = sageattn3(q[:, h:h + 1], k[:, h:h + 1], v[:, h:h + 1], is_causal=True, return_lse=True)
        assert torch.equal(out[:, h:h + 1], one) and torch.equal(lse[:, h:h + 1], one_lse), f"head {h} of {H}"
    h = H // 2
    ref = O.sageattn3_oracle(q[:, h:h + 1].cpu(), k[:, h:h + 1].cpu(), v[:, h:h + 1].cpu(), is_causal=True)
    assert O.cosine(out[:, h:h + 1].cpu(), ref) >= 0.999 and O.rel_l1(out[:, h:h + 1].cpu(), ref) <= 0.01


@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("D", [64, 128])
def test_packed_batch_of_mostly_empty_sequences(cuda_device, D, causal):
    """Sequences without keys, ten or eleven in a row between two that have some (causal: one of these with more queries than keys): several units without
    keys in a row on every SM, between units with keys.  No wait gives up, and every sequence is as it is alone."""
    B, H, Nq = 40, 24, 300
    lens_k = [0] * B
    for i in range(0, B, 13):
        lens_k[i], lens_k[i + (1 if i < 39 else -1)] = 300 + i, 100
    g = torch.Generator(device=cuda_device).manual_seed(1370)
    q = torch.randn(B * Nq, H, D, device=cuda_device, dtype=torch.bfloat16, generator=g)
    k, v = (torch.randn(sum(lens_k), H, D, device=cuda_device, dtype=torch.bfloat16, generator=g) for _ in range(2))
    cu_q = torch.arange(B + 1, dtype=torch.int32, device=cuda_device) * Nq
    cu_k = torch.tensor([0] + lens_k).cumsum(0).to(device=cuda_device, dtype=torch.int32)
    prob = Sage3Problem.for_shape(B, H, H, Nq, max(lens_k), D, torch.bfloat16, cuda_device, is_causal=causal, q_stride=(0, D, H * D), k_stride=(0, D, H * D))
    out = torch.full_like(q, float("nan"))
    rc = _cabi.lib().sage3_fwd_varlen(C.byref(prob.desc), *(t.data_ptr() for t in (cu_q, cu_k, q, k, v, out)), None, prob.ws.buf.data_ptr(),
                                      torch.cuda.current_stream(cuda_device).cuda_stream)
    assert rc == 0 and prob.check_status() == 0
    k0 = 0
    for i, n in enumerate(lens_k):
        mine = out[i * Nq:(i + 1) * Nq]
        if n == 0:
            assert (mine == 0).all(), i
        else:
            alone = sageattn3(q[None, i * Nq:(i + 1) * Nq], k[None, k0:k0 + n], v[None, k0:k0 + n], tensor_layout="NHD", is_causal=causal)[0]
            assert torch.equal(mine, alone), i
        k0 += n


@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("Nk", [1023, 1024, 1025, 1152, 2049])
def test_halves_rolled_and_unrolled_at_64_channels(cuda_device, Nk, causal):
    """Beyond eight key blocks the uniform kernel without a mask has the halves of an item unrolled; the packed variable-length kernel
    has them rolled up to 32: the same bits."""
    H, Nq = 5, 300
    q, k, v = _inputs(cuda_device, 1, H, Nq, Nk, 64, seed=1400 + Nk)
    cu_q, cu_k = (torch.tensor([0, n], dtype=torch.int32, device=cuda_device) for n in (Nq, Nk))
    packed = sageattn_varlen(*(x[0].transpose(0, 1).contiguous() for x in (q, k, v)), cu_q, cu_k, Nq, Nk, is_causal=causal)
    assert torch.equal(sageattn3(q, k, v, is_causal=causal)[0].transpose(0, 1), packed)


@pytest.mark.parametrize("longest", [4096, 4097])
def test_packed_batch_around_the_length_that_unrolls(cuda_device, longest):
    """A packed batch at 64 channels without a mask is walked unrolled, its short sequences too, when the longest has more than 32 key blocks: the
    bits of the sequences alone, some of which are walked the other way."""
    H, lens = 3, [200, longest, 1, 1100]
    g = torch.Generator(device=cuda_device).manual_seed(longest)
    q, k, v = (torch.randn(sum(lens), H, 64, device=cuda_device, dtype=torch.bfloat16, generator=g) for _ in range(3))
    out = sageattn_varlen(q, k, v, *(torch.tensor([0] + lens).cumsum(0).to(device=cuda_device, dtype=torch.int32),) * 2, longest, longest)
    r0 = 0
    for n in lens:
        alone = sageattn3(*(x[None, r0:r0 + n] for x in (q, k, v)), tensor_layout="NHD")[0]
        assert torch.equal(out[r0:r0 + n], alone), n
        r0 += n


@pytest.mark.parametrize("D,tiles,kv_heads", [(128, 101, 40), (128, 100, 40), (64, 76, 40), (64, 77, 40), (64, 78, 40)])
def test_key_tiles_in_runs(cuda_device, D, tiles, kv_heads):
    """Few query blocks and many key tiles: a block of the K kernel walks a run of tiles that ends and begins inside heads, with a ragged last tile: the same
    bits as with one kv head, where every tile has a block of its own.  One head has a key that is not finite in its second tile: it stays there."""
    g = torch.Generator(device=cuda_device).manual_seed(1500 + tiles)
    Nk, group = tiles * 128 - 5, 4
    k, v = (torch.randn(1, kv_heads, Nk, D, device=cuda_device, dtype=torch.bfloat16, generator=g) for _ in range(2))
    q = torch.randn(1, kv_heads * group, 1, D, device=cuda_device, dtype=torch.bfloat16, generator=g)
    for bad in (False, True):
        if bad:
            k[0, 5, 130] = float("nan")
        out = sageattn3(q, k, v, is_causal=True)
        for h in (0, 1, 5, 6, kv_heads - 2, kv_heads - 1):
            few = sageattn3(q[:, h * group:(h + 1) * group], k[:, h:h + 1], v[:, h:h + 1], is_causal=True)
            assert torch.equal(out[:, h * group:(h + 1) * group].nan_to_num(7.0), few.nan_to_num(7.0)), (h, bad)
        assert torch.isfinite(out[:, 6 * group:]).all() and torch.isfinite(out[:, :5 * group]).all()


@pytest.mark.parametrize("D,N,causal", [(128, 5120, False), (64, 3790, True)])
def test_key_tiles_in_runs_with_one_mean_per_head(cuda_device, D, N, causal):
    """One Q mean per head: the K kernel sees one query block per head, however many queries, and walks runs of tiles here too.  The same bits as with
    two kv heads, where every tile (80 or 60 of them) has a block of its own."""
    Hkv, group = 100, 2
    g = torch.Generator(device=cuda_device).manual_seed(1600 + N)
    k, v = (torch.randn(1, Hkv, N, D, device=cuda_device, dtype=torch.float16, generator=g) for _ in range(2))
    q = torch.randn(1, Hkv * group, N, D, device=cuda_device, dtype=torch.float16, generator=g)
    out, lse = sageattn3(q, k, v, is_causal=causal, per_block_mean=False, return_lse=True)
    for h in (0, 51, Hkv - 2):
        few = sageattn3(q[:, h * group:(h + 2) * group], k[:, h:h + 2], v[:, h:h + 2], is_causal=causal, per_block_mean=False, return_lse=True)
        assert torch.equal(out[:, h * group:(h + 2) * group], few[0]) and torch.equal(lse[:, h * group:(h + 2) * group], few[1]), h


@pytest.mark.parametrize("pbm", [True, False])
@pytest.mark.parametrize("D", [64, 128])
def test_key_tiles_in_runs_in_a_packed_batch(cuda_device, D, pbm):
    """A packed batch whose sequences end in a run's first tile, in one of its later tiles or between runs, or have no keys: every sequence as it is
    alone, and a head of it, where every tile has a block of its own."""
    Hkv, group, longest = 8, 2, 51 * 128
    lens = [longest, 1, 127, 128, 129, 0, 255, 256, 257, 384, 385, 640, 6000 + 13]
    n_q = [1, 3, 1, 1, 2, 1, 1, 5, 1, 1, 1, 1, 60]
    B = len(lens)
    g = torch.Generator(device=cuda_device).manual_seed(1700 + D)
    q = torch.randn(sum(n_q), Hkv * group, D, device=cuda_device, dtype=torch.bfloat16, generator=g)
    k, v = (torch.randn(sum(lens), Hkv, D, device=cuda_device, dtype=torch.bfloat16, generator=g) for _ in range(2))
    cu_q, cu_k = (torch.tensor([0] + n).cumsum(0).to(device=cuda_device, dtype=torch.int32) for n in (n_q, lens))
    assert B * Hkv * (longest // 128) >= 3 * torch.cuda.get_device_properties(cuda_device).multi_processor_count
    out = sageattn_varlen(q, k, v, cu_q, cu_k, max(n_q), longest, per_block_mean=pbm)
    q0 = k0 = 0
    for i, (m, n) in enumerate(zip(n_q, lens)):
        mine = out[q0:q0 + m]
        if n == 0:
            assert (mine == 0).all(), i
        else:
            assert torch.equal(mine, sageattn3(q[None, q0:q0 + m], k[None, k0:k0 + n], v[None, k0:k0 + n], tensor_layout="NHD", per_block_mean=pbm)[0]), i
            for h in (0, Hkv - 1):
                one = (q[None, q0:q0 + m, h * group:(h + 1) * group], k[None, k0:k0 + n, h:h + 1], v[None, k0:k0 + n, h:h + 1])
                assert torch.equal(mine[:, h * group:(h + 1) * group], sageattn3(*one, tensor_layout="NHD", per_block_mean=pbm)[0]), (i, h)
        q0, k0 = q0 + m, k0 + n

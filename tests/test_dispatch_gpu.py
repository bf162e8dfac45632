"""The sizes at which the launch path changes: work units of the attention kernel (pairs and single query tiles around
multiples of the SM count), query heads packed into one tile, means formed inside the kernels or by a launch of their own,
output rows on 16- and on 32-byte boundaries, and the host extension against the Python path.  Every head is computed from
its own q, k, v alone, in one order of operations, so the results of different paths must agree bit for bit; against the
oracle the gate is the one of the whole path (cosine >= 0.999, relative L1 <= 1 %)."""
import pytest
import torch

from oracle import sage3_oracle as O
from sageattention_b200 import Sage3Problem, sageattn3, sageattn_varlen

pytestmark = pytest.mark.gpu


def _inputs(device, B, Hq, Hkv, Nq, Nk, D, seed, dtype=torch.bfloat16):
    q, k, v = O.make_inputs(B, Hq, Hkv, Nq, Nk, D, seed=seed, dtype=dtype, k_offset_std=1.0)
    return q.to(device), k.to(device), v.to(device)


@pytest.mark.parametrize("D,causal", [(128, False), (64, True)])
@pytest.mark.parametrize("tiles,half,extra", [(3, 0, -2), (3, 0, 0), (3, 0, 2), (3, 1, 0), (3, 1, 2), (2, 0, -1), (2, 0, 0), (2, 0, 1), (2, 1, 0), (2, 1, 1)])
def test_units_around_the_sm_count(cuda_device, D, causal, tiles, half, extra):
    """Two query tiles per head are one unit, three are two (a pair and a single one).  The units number one round of all SMs, or a round
    and a half, plus `extra`: a round that is not full, a full one, and a second one that is dealt out as single tiles (up to half of the
    SMs) or not."""
    sms = torch.cuda.get_device_properties(cuda_device).multi_processor_count
    units = sms + half * (sms // 2) + extra
    H = units // (tiles - 1)
    assert H * (tiles - 1) == units
    q, k, v = _inputs(cuda_device, 1, H, H, 128 * tiles - 84, 260, D, seed=700 + extra)
    out = sageattn3(q, k, v, is_causal=causal)
    for h in sorted({0, 1, H // 2, H - 2, H - 1}):
        one = sageattn3(q[:, h:h + 1], k[:, h:h + 1], v[:, h:h + 1], is_causal=causal)
        assert torch.equal(out[:, h:h + 1], one), f"head {h} of {H}"


@pytest.mark.parametrize("Nq,Hq,Hkv,Nk,D,causal", [(1, 8, 2, 700, 128, True), (1, 32, 2, 129, 64, False), (9, 14, 2, 128, 128, True),
                                                   (16, 8, 1, 1000, 64, True), (64, 4, 2, 300, 128, True), (65, 4, 2, 300, 128, True),
                                                   (3, 12, 4, 2, 64, True)])
def test_heads_sharing_a_tile(cuda_device, Nq, Hq, Hkv, Nk, D, causal):
    """One to sixteen query heads per kv head, up to eight of them in one tile, at the row counts where a tile is just
    full: the same bits as with the keys and values repeated per query head (no sharing), and the oracle's result."""
    q, k, v = _inputs(cuda_device, 2, Hq, Hkv, Nq, Nk, D, seed=800 + Nq + Hq)
    scale = torch.rand(Hq, generator=torch.Generator().manual_seed(1)) * 0.1 + 0.05
    out, lse = sageattn3(q, k, v, is_causal=causal, sm_scale=scale, return_lse=True)
    g = Hq // Hkv
    rep, rep_lse = sageattn3(q, k.repeat_interleave(g, 1), v.repeat_interleave(g, 1), is_causal=causal, sm_scale=scale, return_lse=True)
    assert torch.equal(out, rep) and torch.equal(lse, rep_lse)
    ref = O.sageattn3_oracle(q.cpu(), k.cpu(), v.cpu(), is_causal=causal, sm_scale=scale)
    assert O.cosine(out.cpu(), ref) >= 0.999 and O.rel_l1(out.cpu(), ref) <= 0.01


@pytest.mark.parametrize("B,Nq,Hq,Hkv,D", [(2, 1, 4, 1, 128), (1, 4, 14, 2, 64), (1, 32, 2, 2, 128), (1, 33, 2, 2, 64), (2, 2, 32, 2, 64),
                                           (1, 4, 8, 1, 128), (1, 5, 8, 1, 128), (3, 1, 60, 60, 64)])
@pytest.mark.parametrize("Nk,causal", [(31, False), (32, True), (33, False), (97, True), (128, True), (129, False), (1300, True)])
def test_few_rows_split_by_keys(cuda_device, B, Nq, Hq, Hkv, D, Nk, causal):
    """Up to 32 rows per kv head: a warp takes 32 keys of a block for all rows.  Row counts around 32, lengths around a
    warp's keys, more units than SMs: the bits of the packed variable-length path, where a warp has rows of its own."""
    q, k, v = _inputs(cuda_device, B, Hq, Hkv, Nq, Nk, D, seed=850 + Nq + Nk)
    out, lse = sageattn3(q, k, v, is_causal=causal, return_lse=True)
    cq, ck = (torch.arange(B + 1, dtype=torch.int32, device=cuda_device) * n for n in (Nq, Nk))
    ref, ref_lse = sageattn_varlen(*(x.transpose(1, 2).flatten(0, 1) for x in (q, k, v)), cq, ck, Nq, Nk, is_causal=causal, return_lse=True)
    assert torch.equal(out.transpose(1, 2).flatten(0, 1), ref) and torch.equal(lse, ref_lse)


@pytest.mark.parametrize("Nk", [128, 1030, 2400])
@pytest.mark.parametrize("D", [64, 128])
def test_few_rows_in_many_units(cuda_device, D, Nk):
    """At most 32 rows per kv head, four units and more per CTA, of 1 to 19 key blocks: one warp of the output group does the work and the
    other three pass units by.  No wait gives up, and the bits are those of the packed variable-length path."""
    B, H, Nq = 8, 80, 2
    q, k, v = _inputs(cuda_device, B, H, H, Nq, Nk, D, seed=870 + Nk)
    prob = Sage3Problem(q, k, v)
    for _ in range(5):
        out = prob.run()
    assert prob.check_status() == 0
    cq, ck = (torch.arange(B + 1, dtype=torch.int32, device=cuda_device) * n for n in (Nq, Nk))
    ref = sageattn_varlen(*(x.transpose(1, 2).flatten(0, 1) for x in (q, k, v)), cq, ck, Nq, Nk)
    assert torch.equal(out.transpose(1, 2).flatten(0, 1), ref)


@pytest.mark.parametrize("Nk", [1, 512, 513, 16384, 16385])
@pytest.mark.parametrize("block_mean", [True, False])
def test_means_inside_and_outside_the_kernels(cuda_device, Nk, block_mean):
    """The K mean is formed by the kernels that use it up to 16 384 keys and by a launch of its own beyond; Q is quantized before
    the means are known unless the LSE or one mean per head is wanted.  All of them against the oracle, and against one another."""
    q, k, v = _inputs(cuda_device, 1, 2, 1, 140, Nk, 64, seed=900 + Nk)
    out = sageattn3(q, k, v, per_block_mean=block_mean)
    out2, lse = sageattn3(q, k, v, per_block_mean=block_mean, return_lse=True)
    assert torch.equal(out, out2)
    ref, ref_lse = O.sageattn3_oracle(q.cpu(), k.cpu(), v.cpu(), per_block_mean=block_mean, return_lse=True)
    assert O.cosine(out.cpu(), ref) >= 0.999 and O.rel_l1(out.cpu(), ref) <= 0.01
    assert (lse.cpu() - ref_lse).abs().max() <= 1e-3       # log2 / exp2 approximations, as in the LSE tests of the whole path


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("heads,Nq", [(8, 8 * 128), (8, 8 * 128 + 1), (1, 128 * 128), (1, 128 * 128 + 1), (8, 16 * 128), (8, 16 * 128 + 1)])
def test_query_blocks_of_a_kv_head_around_one_mma(cuda_device, heads, Nq, D):
    """delta_s takes 128 query blocks of all heads of a kv head at a time, and a smaller tile serves up to 64: 64 and 128 blocks, and
    one more per head."""
    q, k, v = _inputs(cuda_device, 1, heads, 1, Nq, 200, D, seed=1000 + heads)
    out = sageattn3(q, k, v)
    for h in {0, heads - 1}:
        tail = sageattn3(q[:, h:h + 1, -(Nq % 128 or 128):], k, v)         # the last block alone has the same block mean
        assert torch.equal(out[:, h:h + 1, -tail.shape[2]:], tail)


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("Nq,Nk,causal", [(130, n, False) for n in (63, 64, 65, 127, 191, 192, 193, 226)]
                         + [(256, n, True) for n in (160, 192, 193, 255, 256, 257, 288, 319)])
def test_mask_edges_of_half_blocks_and_warps(cuda_device, Nq, Nk, causal, D):
    """Lengths around the 64 keys of a half block and causal shifts around the 32 rows of a warp.  A masked-out key that got
    through would be the only large one: the keys past a row's limit point along its query."""
    q, k, v = _inputs(cuda_device, 1, 2, 2, Nq, Nk, D, seed=950 + Nk)
    if causal:
        rows = torch.arange(Nk, device=q.device) - (Nk - Nq) - 1                  # the query whose first hidden key this is
        hidden = (rows >= 0) & (rows < Nq)
        k[:, :, hidden] += q[:, :, rows[hidden]]
    out = sageattn3(q, k, v, is_causal=causal)
    ref = O.sageattn3_oracle(q.cpu(), k.cpu(), v.cpu(), is_causal=causal)
    assert O.cosine(out.cpu(), ref) >= 0.999 and O.rel_l1(out.cpu(), ref) <= 0.01


@pytest.mark.parametrize("pad", [8, 16])
def test_output_rows_on_16_and_32_byte_boundaries(cuda_device, pad):
    q, k, v = _inputs(cuda_device, 1, 3, 3, 200, 300, 64, seed=1100)
    wide = torch.full((1, 3, 200, 64 + pad), 7.0, dtype=q.dtype, device=cuda_device)
    Sage3Problem(q, k, v, out=wide[..., :64]).run()
    assert torch.equal(wide[..., :64], sageattn3(q, k, v))
    assert (wide[..., 64:] == 7.0).all()


def test_host_extension_and_python_path_agree(cuda_device):
    """Plain tensors go through the host extension; a last dimension that is not contiguous, and a scale given as a tensor, through
    Python.  Two streams have a workspace each."""
    q, k, v = _inputs(cuda_device, 1, 4, 2, 200, 300, 64, seed=1200)
    ref = sageattn3(q, k, v, is_causal=True, sm_scale=0.2)
    qt = q.transpose(2, 3).contiguous().transpose(2, 3)
    assert torch.equal(sageattn3(qt, k, v, is_causal=True, sm_scale=0.2), ref)
    assert torch.equal(sageattn3(q, k, v, is_causal=True, sm_scale=torch.full((4,), 0.2)), ref)
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream(cuda_device) for _ in range(2)]
    outs = []
    for _ in range(4):
        for s in streams:
            with torch.cuda.stream(s):
                outs.append(sageattn3(q, k, v, is_causal=True, sm_scale=0.2))
    torch.cuda.synchronize()
    assert all(torch.equal(o, ref) for o in outs)
    with pytest.raises(ValueError):
        sageattn3(q, k, v, sm_scale=-1.0)
    with pytest.raises(ValueError):
        sageattn3(q, k, v, tensor_layout="BHND")
    with pytest.raises(RuntimeError):
        sageattn3(q.cpu(), k, v)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_scale_of_every_microblock_maximum(cuda_device, dtype):
    """The scale byte and the codes come from a product with 1/6 and an approximate reciprocal of the scale; for every finite positive
    16-bit maximum they have to equal those of the IEEE division and reciprocal.  V is the tensor without smoothing: one maximum
    per microblock of 16 tokens, the other 15 values anywhere below it."""
    from tests._util import canon, read_workspace
    D, groups = 64, 512
    bits = torch.arange(D * groups, dtype=torch.int32) % 0x7F80 if dtype == torch.bfloat16 else torch.arange(D * groups, dtype=torch.int32) % 0x7C00
    peak = bits.to(torch.int16).view(dtype).float().reshape(D, groups)
    g = torch.Generator().manual_seed(5)
    v = peak[..., None] * (2 * torch.rand(D, groups, 16, generator=g) - 1)
    v[..., 3] = peak
    v = v.reshape(D, groups * 16).t().contiguous().to(dtype)[None, None]
    q, k = torch.randn(1, 1, 128, D, generator=g).to(dtype), torch.randn(1, 1, groups * 16, D, generator=g).to(dtype)
    prob = Sage3Problem(q.to(cuda_device), k.to(cuda_device), v.to(cuda_device))
    prob.prepass()
    torch.cuda.synchronize()
    ws, ref = read_workspace(prob), O.prepass(q, k, v)
    assert torch.equal(ws["vt_sf"], ref.vt_sf)
    assert torch.equal(canon(ws["vt_codes"]), canon(ref.vt_codes))


@pytest.mark.parametrize("what", ["k_nan", "q_inf", "delta_overflow"])
@pytest.mark.parametrize("Nq,Hq,Hkv,D", [(1, 32, 8, 128), (1, 4, 4, 64), (9, 14, 2, 128), (40, 6, 2, 64), (4, 18, 2, 128), (2, 32, 4, 64),
                                              (1, 400, 200, 64), (1, 1000, 500, 64)])
def test_non_finite_values_stay_with_their_head(cuda_device, Nq, Hq, Hkv, D, what):
    """Heads that share a tile share the operand that adds delta_s, where 0 x NaN and 0 x Inf are NaN.  One query head, or one kv
    head, of sequence 1 is not finite (a NaN key, an Inf query, an fp16 delta_s that overflows): sequence 0 and the other heads
    get the bits of a call without it, and the head itself what the packed variable-length path, one head per tile, gives it.
    (400 kv heads: more notes than a block has threads; 1 000: more than one block clears.)"""
    dtype = torch.float16 if what == "delta_overflow" else torch.bfloat16
    Nk, B, g = 400, 2, Hq // Hkv
    q, k, v = _inputs(cuda_device, B, Hq, Hkv, Nq, Nk, D, seed=1300 + Nq + Hq, dtype=dtype)
    good = sageattn3(q, k, v, return_lse=True)
    if what == "k_nan":
        k[1, 0, 5, 3] = float("nan")
    elif what == "q_inf":
        q[1, min(1, g - 1), 0, 3] = float("inf")
    else:
        q[1, min(1, g - 1)] = 6.0e4
        k[1, 0, 5] = 200.0
    out, lse = sageattn3(q, k, v, return_lse=True)
    cq, ck = (torch.arange(B + 1, dtype=torch.int32, device=cuda_device) * n for n in (Nq, Nk))
    ref, ref_lse = sageattn_varlen(*(x.transpose(1, 2).flatten(0, 1) for x in (q, k, v)), cq, ck, Nq, Nk, return_lse=True)
    assert not torch.isfinite(ref_lse).all() or (ref == 0).all(-1).any()          # the values do reach that head
    healthy = torch.ones(B, Hq, dtype=torch.bool, device=cuda_device)
    healthy[1, :g] = False                                                        # (in the third case their K differs)
    assert torch.equal(out[healthy], good[0][healthy]) and torch.equal(lse[healthy], good[1][healthy])
    assert torch.equal(out.transpose(1, 2).flatten(0, 1).nan_to_num(7.0), ref.nan_to_num(7.0))
    assert torch.equal(lse.nan_to_num(7.0), ref_lse.nan_to_num(7.0))


def test_threads_on_one_stream_share_a_workspace(cuda_device):
    """Several threads, all on the default stream and so on one workspace, through the host extension, the Python path (a scale per
    head) and the packed entry; more units than SMs, so that a work counter another call has used up would leave rows unwritten."""
    import threading
    N, H = 260, 160
    cu = torch.tensor([0, N], dtype=torch.int32, device=cuda_device)
    per_head = torch.full((H,), 0.2, device=cuda_device)

    def call(i, q, k, v):
        if i == 2:
            return sageattn_varlen(*(x[0].transpose(0, 1) for x in (q, k, v)), cu, cu, N, N, sm_scale=0.2).transpose(0, 1)[None]
        return sageattn3(q, k, v, sm_scale=per_head if i == 1 else 0.2)
    inputs = [_inputs(cuda_device, 1, H, H, N, N, 64, seed=1600 + i) for i in range(3)]
    refs = [call(i, *x) for i, x in enumerate(inputs)]
    torch.cuda.synchronize()
    outs, start = [[] for _ in inputs], threading.Barrier(len(inputs))

    def work(i):
        start.wait()
        for _ in range(30):
            outs[i].append(call(i, *inputs[i]))
    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(inputs))]
    [t.start() for t in threads]
    [t.join() for t in threads]
    torch.cuda.synchronize()
    for i, ref in enumerate(refs):
        assert len(outs[i]) == 30 and all(torch.equal(o, ref) for o in outs[i])


@pytest.mark.parametrize("maxima", [(), (230, 230)])
def test_varlen_output_keeps_the_strides_of_q(cuda_device, maxima):
    """A packed q that is a permuted view, or a slice of a wider tensor: the output is laid out like torch.empty_like(q), whether the
    maxima are given (host extension) or not (Python path)."""
    lens = torch.tensor([0, 70, 300], dtype=torch.int32, device=cuda_device)
    q, k, v = (x[0].transpose(0, 1) for x in _inputs(cuda_device, 1, 4, 2, 300, 300, 64, seed=1400))
    ref = sageattn_varlen(q.contiguous(), k, v, lens, lens, *maxima)
    assert ref.is_contiguous()
    wide = torch.empty(300, 7, 64, dtype=q.dtype, device=cuda_device)
    wide[:, :4] = q
    for view in (q, wide[:, :4]):
        out = sageattn_varlen(view, k, v, lens, lens, *maxima)
        assert out.stride() == torch.empty_like(view).stride()
        assert torch.equal(out, ref)


def test_scale_that_is_zero_in_fp32_is_refused(cuda_device):
    """1e-60 is positive but 0 as the 32-bit scale of the descriptor, where 0 stands for the default; 1e-38 is a scale."""
    q, k, v = _inputs(cuda_device, 1, 2, 2, 100, 100, 64, seed=1500)
    packed = [x[0].transpose(0, 1) for x in (q, k, v)]
    cu = torch.tensor([0, 100], dtype=torch.int32, device=cuda_device)
    for scale in (1e-60, 0.0, float("nan")):
        with pytest.raises(ValueError):
            sageattn3(q, k, v, sm_scale=scale)
        with pytest.raises(ValueError):
            sageattn_varlen(*packed, cu, cu, 100, 100, sm_scale=scale)
    assert not torch.equal(sageattn3(q, k, v, sm_scale=1e-38), sageattn3(q, k, v))


@pytest.mark.parametrize("per_head", [False, True])
def test_a_captured_call_keeps_its_workspace(cuda_device, per_head):
    """A functional call captured on a stream that has made calls before: a larger call replaces the stream's workspace, and
    the memory it had goes to other tensors.  Replays write to none of them and still give the call's result."""
    q, k, v = _inputs(cuda_device, 1, 8, 8, 500, 500, 64, seed=1700)
    big = _inputs(cuda_device, 1, 32, 32, 1000, 1000, 64, seed=1701)
    scale = torch.full((8,), 0.2, device=cuda_device) if per_head else 0.2              # through Python / the host extension
    s = torch.cuda.Stream(cuda_device)
    torch.cuda.synchronize()
    with torch.cuda.stream(s):
        ref = sageattn3(q, k, v, sm_scale=scale)
        s.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s):
            out = sageattn3(q, k, v, sm_scale=scale)
        big_ref = sageattn3(*big)
        fill = [torch.full((1 << 20,), 7, dtype=torch.uint8, device=cuda_device) for _ in range(64)]
        for _ in range(3):
            out.zero_()
            g.replay()
        again = sageattn3(*big)
    torch.cuda.synchronize()
    assert torch.equal(out, ref) and torch.equal(again, big_ref)
    assert all((f == 7).all() for f in fill)

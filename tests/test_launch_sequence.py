"""CPU tests of what the library's host code enqueues: its own object files, linked with a CUDA runtime that records the launches
instead of making them (tests/fake_cudart.cpp)."""
import ctypes as C
import os
import pathlib
import subprocess
import threading

import pytest

from sageattention_b200 import _cabi, build

WS = 1 << 20              # "device" addresses: never dereferenced by host code


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    objs = [build.PKG / "build" / (s + ".o") for s in build.SOURCES]
    srcs = [build.CSRC / s for s in build.SOURCES + build.HEADERS]
    tmp = tmp_path_factory.mktemp("fake")
    if not all(o.exists() for o in objs) or max(s.stat().st_mtime for s in srcs) > min(o.stat().st_mtime for o in objs):
        objs = [tmp / (s + ".o") for s in build.SOURCES]
        procs = [subprocess.Popen(["nvcc", *build.NVCC_FLAGS, "-c", str(build.CSRC / s), "-o", str(o)]) for s, o in zip(build.SOURCES, objs)]
        assert [p.wait() for p in procs] == [0] * len(procs)
    so = tmp / "libsage3_fake.so"
    cuda = pathlib.Path(os.environ.get("CUDA_HOME", "/usr/local/cuda"))
    subprocess.check_call(["g++", "-O1", "-std=c++17", "-fPIC", "-shared", "-Wl,-Bsymbolic", f"-isystem{cuda / 'include'}",
                           str(pathlib.Path(__file__).with_name("fake_cudart.cpp")), *map(str, objs), "-o", str(so), "-lpthread"])
    lib = C.CDLL(str(so))
    lib.fake_log.restype = lib.fake_kernels.restype = C.c_char_p
    return lib


def _desc(**kw):
    d = _cabi.Sage3Desc()
    base = dict(B=1, Hq=4, Hkv=2, Nq=300, Nk=700, D=64, dtype=_cabi.SAGE3_BF16, is_causal=0, per_block_mean=1)
    base.update(kw)
    for k, v in base.items():
        setattr(d, k, v)
    n = max(base["Nq"], base["Nk"])
    for name in ("q_stride", "k_stride", "v_stride", "o_stride"):
        setattr(d, name, (C.c_int64 * 3)(base["Hq"] * n * base["D"], n * base["D"], base["D"]))
    return d


def _fwd(lib, d, ws=WS, lse=None):
    p = C.c_void_p
    return lib.sage3_fwd(C.byref(d), p(1 << 12), p(1 << 13), p(1 << 14), p(ws), p(1 << 15), p(lse), None)


def _varlen(lib, d, ws=WS, lse=None):
    p = C.c_void_p
    return lib.sage3_fwd_varlen(C.byref(d), p(1 << 10), p(1 << 11), p(1 << 12), p(1 << 13), p(1 << 14), p(1 << 15), p(lse), p(ws), None)


def _carried(lib, d):
    p, carry = C.c_void_p, _cabi.Sage3Carry()
    carry.o_out, carry.m_out, carry.l_out = (1 << 20,) * 3
    return lib.sage3_attn_fwd_carry(C.byref(d), p(WS), C.byref(carry), None, None, None)


def _log(lib):
    return [line.split(":") for line in lib.fake_log().decode().splitlines()]


@pytest.mark.parametrize("call", [_fwd, _varlen])
@pytest.mark.parametrize("kw,lse", [({}, None), (dict(per_block_mean=0, Nk=20000), 1 << 16)])
def test_calls_of_two_threads_on_one_workspace_do_not_interleave(fake, call, kw, lse):
    """The kernels of a call hand their results on through the workspace: another call that uses it may come before or after all
    of them only.  (Every launch pauses, so that threads that may interleave do.)"""
    fake.fake_start(-1, 2000)
    start, rcs = threading.Barrier(3), []

    def work():
        start.wait()
        for _ in range(3):
            rcs.append(call(fake, _desc(**kw), lse=lse))
    threads = [threading.Thread(target=work) for _ in range(3)]
    [t.start() for t in threads]
    [t.join() for t in threads]
    log = _log(fake)
    assert rcs == [0] * 9 and len(log) % 9 == 0
    per_call = len(log) // 9
    assert per_call >= 3
    for i in range(0, len(log), per_call):
        assert len({entry[0] for entry in log[i:i + per_call]}) == 1, log[i:i + per_call]


CALLS = [(_fwd, {}, None), (_fwd, {}, 1 << 16), (_fwd, dict(Nk=20000), None), (_fwd, dict(Nk=20000, Nq=20000, per_block_mean=0), None),
         (_varlen, dict(per_block_mean=0, Nk=20000), 1 << 16)]


@pytest.mark.parametrize("call,kw,lse", CALLS)
def test_a_refused_launch_is_reported_and_ends_the_call(fake, call, kw, lse):
    """Whichever launch of a call the runtime refuses: the call returns SAGE3_E_CUDA, enqueues nothing after it (the kernels behind
    it would work on what an earlier call left), and leaves no error behind for whoever asks the runtime next."""
    fake.fake_start(-1, 0)
    assert call(fake, _desc(**kw), lse=lse) == 0
    n = len(_log(fake))
    for i in range(n):
        fake.fake_start(i, 0)
        assert call(fake, _desc(**kw), lse=lse) == -7, i
        log = _log(fake)
        assert len(log) == i + 1 and log[-1][-1] == "refused", log
        assert fake.fake_last_error() == 0, i


def _attn(lib, d):
    p = C.c_void_p
    return lib.sage3_attn_fwd(C.byref(d), p(WS), p(1 << 15), None, None)


def _attn_parts(lib, d):
    p, parts = C.c_void_p, _cabi.Sage3Parts()
    parts.parts, parts.rows_per_part = 2, (d.Nq + 1) // 2
    parts.base[0] = parts.base[1] = 1 << 15
    return lib.sage3_attn_fwd_parts(C.byref(d), p(WS), C.byref(parts), None, None)


@pytest.mark.parametrize("call,kw", [
    (_attn, {}), (_attn, dict(Nk=9000)), (_attn, dict(Nq=1000, Nk=9192, Hq=32, is_causal=1, D=128)),      # ... tiles shared
    (_attn, dict(Nq=1, Hq=32, Nk=9000)), (_carried, dict(Nk=9000)), (_attn_parts, dict(Nq=1000, Nk=9192, Hq=32, D=128)), (_attn_parts, dict(Nk=9000))])
def test_attention_on_its_own_is_one_memset_and_one_kernel(fake, call, kw):
    """What the kernel wants cleared lies in one piece: each further stream operation takes longer than a microsecond."""
    fake.fake_start(-1, 0)
    assert call(fake, _desc(**kw)) == 0
    names = [entry[1] for entry in _log(fake)]
    assert len(names) == 2 and names[0] == "memset" and "attn_fwd" in names[1], names


def test_shared_memory_is_asked_for_once_per_kernel(fake):
    """Calls that between them launch every attention and every K kernel of the library: in a second round no kernel's attributes are set again (that is a call into the
    runtime for every launch, paid by the shortest calls)."""
    full = [dict(Nk=700), dict(Nk=3000), dict(Nq=128 * 33),                                # whole tiles; many query blocks
            dict(Hq=32, Nq=1000, Nk=9192),                                                 # tiles shared
            dict(Hq=2, Hkv=1, Nq=128 * 17, Nk=60000), dict(Hq=4, Hkv=1, Nq=128 * 17, Nk=60000)]      # 34 and 68 query blocks over many key tiles
    few = [dict(Nq=16, Hq=16), dict(Nq=1, Hq=8), dict(Nq=1, Hq=66, Hkv=1),                 # heads that share a tile, of 8, 4 and 66 query blocks
           dict(B=8, Nq=1, Hq=32, Hkv=8, Nk=20000), dict(B=8, Nq=1, Hq=8, Hkv=8, Nk=20000),      # many key tiles
           dict(Nq=1, Hq=33, Hkv=1, Nk=60000), dict(Nq=1, Hq=66, Hkv=1, Nk=60000)]
    kernels = set()
    for _ in range(2):
        fake.fake_start(-1, 0)
        for dtype in (_cabi.SAGE3_BF16, _cabi.SAGE3_FP16):
            for D in (64, 128):
                for causal in (0, 1):
                    kw = dict(dtype=dtype, D=D, is_causal=causal)
                    assert [_fwd(fake, _desc(**kw, **c)) for c in full + few] == [0] * (len(full) + len(few))
                    assert [f(fake, _desc(**kw, Nk=n)) for f in (_varlen, _carried) for n in (700, 3000, 9000)] == [0] * 6
        kernels |= {entry[1] for entry in _log(fake) if "attn_fwd" in entry[1] or "quant_k_delta" in entry[1]}
    assert kernels == {k for k in fake.fake_kernels().decode().split() if "attn_fwd" in k or "quant_k_delta" in k} and len(kernels) == 88
    assert fake.fake_attributes() == 0


@pytest.mark.parametrize("call,Nk,causal,D,rolled", [(_fwd, 1024, 0, 64, 1), (_fwd, 1025, 0, 64, 0), (_fwd, 9000, 1, 64, 1), (_fwd, 9000, 0, 128, 1),
                                                     (_varlen, 4096, 0, 64, 1), (_varlen, 4097, 0, 64, 0), (_varlen, 9000, 1, 64, 1), (_varlen, 9000, 0, 128, 1),
                                                     (_carried, 700, 0, 128, 0), (_carried, 9000, 1, 128, 0), (_carried, 700, 1, 64, 1), (_carried, 9000, 0, 64, 1)])
def test_halves_are_unrolled_where_that_is_faster(fake, call, Nk, causal, D, rolled):
    """The attention kernel's last template argument: its halves rolled, except at 64 channels without a mask over many key blocks, and with
    carried state at 128 channels."""
    fake.fake_start(-1, 0)
    assert call(fake, _desc(Nk=Nk, Nq=Nk, is_causal=causal, D=D)) == 0
    name = [entry[1] for entry in _log(fake) if "attn_fwd" in entry[1]][0]
    assert f"ELb{rolled}EEEv" in name, name


@pytest.mark.parametrize("D,tiles,blocks,kernel,rows", [
    (128, 148, 1, "", 64), (128, 148, 64, "", 64), (128, 148, 65, "", 128), (128, 149, 32, "_run", 32), (128, 149, 33, "_run", 64), (128, 149, 64, "_run", 64),
    (128, 149, 65, "", 128), (128, 4000, 8, "_run", 32), (128, 4000, 65, "", 128),
    (64, 148, 32, "", 64), (64, 148, 128, "", 128), (64, 149, 32, "", 64), (64, 149, 33, "_run", 64), (64, 296, 64, "_run", 64), (64, 296, 65, "_run", 128), (64, 297, 33, "", 64),
    (64, 297, 128, "", 128), (64, 444, 32, "", 64), (64, 444, 64, "", 64), (64, 444, 65, "", 128), (64, 445, 1, "_run", 32), (64, 445, 32, "_run", 32), (64, 445, 64, "_run", 64),
    (64, 445, 128, "_run", 128), (64, 445, 129, "", 128), (64, 4000, 8, "_run", 32)])
def test_which_kernel_takes_k(fake, D, tiles, blocks, kernel, rows):
    """A block of the K kernel has one tile or walks a run of them, by the number of key tiles per SM (148 here) and of query blocks of all query heads of a kv head (one per
    head with one Q mean); the rows or columns that it has for these."""
    name = f"quant_k_delta{kernel}_kernelI13__nv_bfloat16Li{D}ELi{rows}E"
    for kw in (dict(Nq=1, Hq=blocks), dict(Nq=128 * blocks - 5, Hq=1), dict(Nq=300, Hq=blocks, per_block_mean=0)):
        fake.fake_start(-1, 0)
        assert _fwd(fake, _desc(**dict(dict(B=1, Hkv=1, Nk=128 * tiles, D=D), **kw))) == 0
        assert [entry[1] for entry in _log(fake) if "quant_k_delta" in entry[1]][0].find(name) >= 0, kw


def test_a_launch_of_too_many_blocks_is_refused():
    """All pieces of the first pre-pass kernel are one grid: their number, not that of one kind, has to stay below 2^31."""
    d = _desc(B=60000, Hq=1, Hkv=1, Nq=128, Nk=6000000)       # 2.8e9 tiles of V
    assert _cabi.lib().sage3_workspace_bytes(C.byref(d)) == 0
    assert _cabi.lib().sage3_workspace_layout(C.byref(d), C.byref(_cabi.Sage3Workspace())) == -8
    d = _desc(B=60000, Hq=1, Hkv=1, Nq=128, Nk=3000000)
    assert _cabi.lib().sage3_workspace_bytes(C.byref(d)) > 0

"""What the packed attention entry points accept and refuse before they launch anything (CPU)."""
import ctypes
import os
import subprocess
import sys
from ctypes import c_float, c_int, c_int64, c_void_p

import pytest

import pytest
import torch

from dhellam_b200 import kernels as K


def _backward_with(lengths, heads):
    """Error text of a packed backward over null operands: the operands are the last thing that is looked at before a launch."""
    cu = [0]
    for n in lengths:
        cu.append(cu[-1] + n)
    off = (c_int * len(cu))(*cu)
    p_int = ctypes.POINTER(c_int)
    fn = K.proto("dh_attn_bwd_packed", [c_void_p] * 10 + [ctypes.POINTER(c_int64), c_int, p_int, p_int, c_int, c_int, c_int, c_int, c_int,
                                                          c_int, c_int, c_float, c_int, c_void_p])
    rc = fn(*[0] * 10, (c_int64 * 24)(*[heads * 128, heads * 128, 128] * 8), len(lengths), off, off, cu[-1], cu[-1], max(lengths), heads,
            heads, 128, 1, 1.0, 0, 0)
    assert rc != 0
    return K.lib().dh_last_error_string().decode()


def test_the_row_limit_of_the_backward_holds_per_sequence():
    """64 heads and 2^21 tokens in documents of unequal length: 2^27 rows in all, at most 2^25 in one sequence."""
    lengths = [2 ** 19, 2 ** 19 - 7, 2 ** 18, 2 ** 19, 2 ** 18 + 7]
    assert 64 * sum(lengths) > 2 ** 26 > 64 * max(lengths)
    assert "2^26" not in _backward_with(lengths, 64)
    assert "2^26" in _backward_with([2 ** 20 + 1, 5], 64)


def _operands(tq=50, tk=50):
    bf = lambda t, h: torch.zeros(t, h, 128, dtype=torch.bfloat16)
    return dict(q=bf(tq, 2), k=bf(tk, 1), v=bf(tk, 1), dout=bf(tq, 2), out=bf(tq, 2), lse=torch.zeros(2, 2, 30),
                dq=bf(tq, 2), dk=bf(tk, 1), dv=bf(tk, 1))


BAD = {"fp16": lambda t: t.half(), "fp32": lambda t: t.double() if t.dtype == torch.float32 else t.float(), "short": lambda t: t[:49],
       "heads": lambda t: t.repeat(1, 2, 1), "columns": lambda t: torch.cat([t, t], 2)[:, :, ::2]}


# (the shape of the statistics is looked at by the caller)
@pytest.mark.parametrize("which,how", [(w, h) for w in ("q", "k", "v", "dout", "out", "lse") for h in BAD if w != "lse" or h.startswith("fp")])
def test_operands_that_the_kernels_would_misread_are_refused(which, how):
    """Other types, too few rows, other heads or strided columns: the kernels see addresses and strides only."""
    from dhellam_b200.ops.attention_native import attn_bwd_packed, attn_fwd_packed
    o = _operands()
    o[which] = BAD[how](o[which])
    cu = [0, 20, 50]
    if which in ("q", "k", "v") and not (which == "q" and how == "heads"):     # four query heads on one KV head are fine
        with pytest.raises(AssertionError):
            attn_fwd_packed(o["q"], o["k"], o["v"], cu, cu, 30, True, None)
    with pytest.raises(AssertionError):
        attn_bwd_packed(o["dout"], o["q"], o["k"], o["v"], o["out"], o["lse"], o["dq"], o["dk"], o["dv"], cu, cu, True, None)


@pytest.mark.parametrize("tq,tk", [(50, 0), (0, 50), (0, 0)])
def test_batches_without_any_key_or_query_give_zeros(tq, tk):
    """As the empty sequences of a batch that has others: no probability, no gradient."""
    from dhellam_b200.ops.attention_native import attn_bwd_packed, attn_fwd_packed
    o = {n: torch.full_like(t, float("nan")) for n, t in _operands(tq, tk).items()}
    cq, ck = [0, tq * 2 // 5, tq], [0, tk * 2 // 5, tk]
    if tk == 0:
        for max_q in (30, 40):
            out, lse = attn_fwd_packed(o["q"], o["k"], o["v"], cq, ck, max_q, True, None)
            assert out.shape == o["q"].shape and not out.any() and lse.shape == (2, 2, max_q) and (lse == float("-inf")).all()
    attn_bwd_packed(o["dout"], o["q"], o["k"], o["v"], o["out"], o["lse"], o["dq"], o["dk"], o["dv"], cq, ck, True, None)
    assert not any(o[n].any() for n in ("dq", "dk", "dv"))


def _launches(lengths, causal=1):
    cu = [0]
    for n in lengths:
        cu.append(cu[-1] + n)
    off, p_int = (c_int * len(cu))(*cu), ctypes.POINTER(c_int)
    return K.proto("dh_attn_packed_launches", [c_int, p_int, p_int, c_int])(len(lengths), off, off, causal)


def test_a_long_sequence_is_cut_into_launches():
    """A tile's index fits its field of the launch's table whatever the length: 2^24 rows are 131072 tiles, 768 to a launch."""
    assert _launches([2 ** 24, 100]) == 171


@pytest.mark.parametrize("lengths,most", [([1024] * 300, 5), ([128] * 1024, 8), ([64] * 129, 2), ([0] * 500 + [4096] * 24, 5),
                                          ([17 + 31 * (i % 97) for i in range(640)], 13), ([8192] * 64, 6)])
def test_many_sequences_take_about_as_few_launches_as_their_tables_allow(lengths, most):
    """At most 768 tiles of 128 sequences to a launch; a batch of more sequences is divided by length before its tiles are sorted."""
    tiles = sum((n + 127) // 128 for n in lengths)
    assert max(-(-tiles // 768), -(-sum(n > 0 for n in lengths) // 128)) <= _launches(lengths) <= most


def test_a_failed_host_allocation_is_an_error_code():
    """The list of tiles of 2^30 rows does not fit what the process may still allocate: the C entry point answers, it does not abort."""
    code = """
import resource
from test_attention_packed_limits import _launches
assert _launches([1000]) == 1
used = int(open("/proc/self/statm").read().split()[0]) * resource.getpagesize()
resource.setrlimit(resource.RLIMIT_AS, (used + (64 << 20), -1))
assert _launches([2 ** 30]) == -2                # out of memory, as a CUDA error code
"""
    env = dict(os.environ, PYTHONPATH=os.pathsep.join(sys.path))
    run = subprocess.run([sys.executable, "-c", code], env=env, capture_output=True, text=True)
    assert run.returncode == 0, run.stderr

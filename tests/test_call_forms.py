"""Which form of the attention kernel a call takes: `sage_attention_form` is the function the launch asks."""
import ctypes

import pytest

from sageattention import _native


def form(b, hq, hkv, nq, nk, packed_q=0, causal=0, plain=1, sms=148):
    out = (ctypes.c_int * 4)()
    assert _native.load().sage_attention_form(b, hq, hkv, nq, nk, packed_q, causal, plain, sms, out) == 4
    return tuple(out)                      # query tiles per CTA, shares of the keys, folded heads, tests


@pytest.mark.parametrize("call,want", [
    ((1, 48, 48, 47520, 47520), (2, 1, 1, 0)),       # the headline call
    ((1, 48, 48, 4096, 4096), (1, 1, 1, 0)),
    # up to eight key tiles: one query tile per CTA, whatever the rounds rule says of the queries
    ((1, 48, 48, 288, 288), (1, 1, 1, 0)),
    ((1, 40, 40, 16384, 512), (1, 1, 1, 0)),
    ((1, 40, 40, 16384, 1024), (1, 1, 1, 0)),
    ((1, 40, 40, 16384, 1025), (2, 1, 1, 0)),
    # heads of a group share query tiles where those are mostly empty
    ((2, 8, 2, 4, 300), (1, 1, 4, 0)),
    ((1, 8, 2, 128, 300), (1, 1, 1, 0)),             # full tiles
])
def test_fixed_length_calls(call, want):
    assert form(*call) == want


def test_negligible_tile_tests():
    assert form(1, 48, 48, 4096, 4096, plain=0)[3] == 1
    assert form(1, 48, 48, 4096, 1024, plain=0)[3] == 0              # short key loops have none
    assert form(4, 48, 48, 4096, 4096, packed_q=9000, plain=0)[3] == 0
    assert form(1, 48, 48, 4096, 4096, causal=1, plain=0)[3] == 1


@pytest.mark.parametrize("n_seq,longest,tokens,heads,causal,keys,tiles", [
    # batches on which both shapes were timed on a 148-SM part, whole call, one / two tiles per CTA in us
    (64, 128, 64 * 128, 92, 0, 128, 1),              # 430 / 626: the second tile of every CTA would be empty
    (128, 300, 128 * 300, 20, 0, 300, 1),            # 603 / 754
    (32, 512, 32 * 512, 46, 0, 512, 1),              # 491 / 532
    (16, 1024, 16 * 1024, 46, 0, 1024, 1),           # 644 / 680
    (8, 2048, 8 * 2048, 96, 0, 2048, 1),             # 2002 / 2037
    (8, 3100, 8 * 3100, 48, 0, 3100, 1),             # 2139 / 2208
    (11, 8192, 36124, 48, 0, 8192, 1),               # 4152 / 4152
    (5, 4100, 5 * 4100, 37, 0, 4100, 1),             # 1707 / 1732
    (2, 8192, 2 * 8192, 48, 0, 8192, 2),             # 3066 / 2992
    (5, 8192, 26705, 32, 0, 8192, 2),                # 2580 / 2554
    (3, 8192, 3 * 8192, 8, 0, 8192, 1),              # 792 / 831: five rounds
    (2, 8192, 2 * 8192, 48, 1, 8192, 1),             # 1754 / 1778
    (2, 8192, 2 * 8192, 48, 0, 1024, 1),             # short key loops take one tile as in every other call
])
def test_packed_batches(n_seq, longest, tokens, heads, causal, keys, tiles):
    assert form(n_seq, heads, heads, longest, keys, packed_q=tokens, causal=causal) == (tiles, 1, 1, 0)


def test_packed_batches_without_a_work_list_take_one_tile():
    assert form(513, 96, 96, 8192, 8192, packed_q=513 * 8192)[0] == 1


def test_bad_arguments():
    out = (ctypes.c_int * 4)()
    f = _native.load().sage_attention_form
    assert f(1, 3, 2, 8, 8, 0, 0, 0, 148, out) == _native.SAGE_E_ARG
    assert f(1, 2, 2, 8, 8, 0, 0, 0, 0, out) == _native.SAGE_E_ARG
    assert f(1, 2, 2, 8, 8, -1, 0, 0, 148, out) == _native.SAGE_E_ARG
    assert f(1, 2, 2, 8, 8, 0, 0, 0, 148, None) == _native.SAGE_E_ARG

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


def test_bad_arguments():
    out = (ctypes.c_int * 4)()
    f = _native.load().sage_attention_form
    assert f(1, 3, 2, 8, 8, 0, 0, 0, 148, out) == _native.SAGE_E_ARG
    assert f(1, 2, 2, 8, 8, 0, 0, 0, 0, out) == _native.SAGE_E_ARG
    assert f(1, 2, 2, 8, 8, -1, 0, 0, 148, out) == _native.SAGE_E_ARG
    assert f(1, 2, 2, 8, 8, 0, 0, 0, 148, None) == _native.SAGE_E_ARG

"""The rules on sizes that pick a kernel, called in the built library (no GPU needed)."""
import ctypes as C

import pytest

from nvfuserexamples_b200 import capi


def pair_pays(sms, B, H, S_q, S_k, packed_rows=0, lengths=True):
    fn = capi.load()["_ZN4fmha13fwd_pair_paysElllllbl"]   # fmha::fwd_pair_pays(int64_t x 5, bool, int64_t)
    fn.argtypes, fn.restype = [C.c_int64] * 5 + [C.c_bool, C.c_int64], C.c_bool
    return fn(sms, B, H, S_q, S_k, lengths, packed_rows)


def test_two_tile_rule():
    assert pair_pays(148, 4, 16, 2048, 2048)       # 4 sequences of 16 heads: the shape the kernel was built for
    assert not pair_pays(148, 4, 16, 2048, 256)    # two key steps
    assert not pair_pays(148, 4, 16, 512, 2048)    # fewer than two query tiles per multiprocessor
    assert not pair_pays(148, 50, 4, 384, 384)     # three query tiles per head


def test_two_tile_rule_without_a_multiprocessor_count():
    """The number of multiprocessors is 0 where its query failed: the one-tile kernel, not a division by zero."""
    assert not pair_pays(0, 4, 16, 2048, 2048)


@pytest.mark.parametrize("B,H,max_len,rows,pairs", [
    (10, 8, 512, 153, False), (20, 4, 512, 40, False),    # small grids of short sequences: a tile has its SM to itself
    (10, 8, 512, 307, False),                             # pairs would need a second round, tiles do not
    (10, 8, 512, 512, True), (10, 8, 512, 700, True),     # full, and a buffer with rows to spare
    (64, 16, 512, 102, True), (16, 16, 2048, 50, True),   # large grids of short sequences: pairs spare the empty CTAs
    (4, 16, 2048, 409, True),
])
def test_two_tile_rule_sees_how_full_a_packed_batch_is(B, H, max_len, rows, pairs):
    assert pair_pays(148, B, H, max_len, max_len)
    assert pair_pays(148, B, H, max_len, max_len, B * rows) == pairs


def test_two_tile_rule_on_one_round():
    """Pairs that have a multiprocessor each, of long keys and one length; with a pair too many, shorter keys or lengths it is not taken."""
    assert pair_pays(148, 1, 16, 2048, 2048, lengths=False)        # 256 tiles, 128 pairs
    assert not pair_pays(148, 1, 16, 2048, 2048, lengths=True)
    assert not pair_pays(148, 2, 16, 1024, 1023, lengths=False)
    assert not pair_pays(148, 1, 8, 2048, 2048, lengths=False)     # 128 tiles: each has one of its own
    assert not pair_pays(148, 1, 15, 2432, 2432, lengths=False)    # 150 pairs


def chain_pays(sms, tiles, S_k, keyadd, dropout):
    fn = capi.load()["_ZN4fmha14fwd_chain_paysElllbb"]   # fmha::fwd_chain_pays(int64_t x 3, bool, bool)
    fn.argtypes, fn.restype = [C.c_int64] * 3 + [C.c_bool] * 2, C.c_bool
    return fn(sms, tiles, S_k, keyadd, dropout)


def test_rule_of_the_kernel_that_goes_from_tile_to_tile():
    assert chain_pays(148, 593, 256, False, False) and not chain_pays(148, 592, 256, False, False)   # one tile more than are resident
    assert chain_pays(148, 593, 384, True, False) and not chain_pays(148, 593, 384, False, False)    # six key steps want three rounds
    assert chain_pays(148, 1776, 384, False, False) and not chain_pays(148, 9999, 385, True, False)
    assert chain_pays(148, 1480, 640, False, True) and not chain_pays(148, 1479, 640, False, True)   # dropout: two and a half
    assert chain_pays(148, 1776, 640, True, True) and not chain_pays(148, 1775, 640, True, True)
    assert not chain_pays(148, 9999, 641, False, True)
    assert not chain_pays(0, 0, 64, False, False)


def test_rule_of_the_kernel_that_goes_from_tile_to_tile_without_lengths():
    """One length of four whole key steps: not where the second round is nearly full."""
    fn = capi.load()["_ZN4fmha14fwd_chain_paysElllbbb"]   # fmha::fwd_chain_pays(int64_t x 3, bool x 3)
    fn.argtypes, fn.restype = [C.c_int64] * 3 + [C.c_bool] * 3, C.c_bool
    assert fn(148, 1006, 256, False, False, False) and not fn(148, 1007, 256, False, False, False)
    assert not fn(148, 1184, 241, False, False, False) and fn(148, 1185, 256, False, False, False)
    assert fn(148, 1184, 240, False, False, False) and fn(148, 1184, 256, False, False, True) and fn(148, 1184, 256, True, False, False)
    assert not fn(148, 1184, 256, False, True, False) and not fn(148, 592, 64, False, False, False)


def one_kv(D, heads, S_q, S_k):
    fn = capi.load()["_ZN4fmha10bwd_one_kvEilii"]   # fmha::bwd_one_kv(int, int64_t, int, int)
    fn.argtypes, fn.restype = [C.c_int, C.c_int64, C.c_int, C.c_int], C.c_bool
    return fn(D, heads, S_q, S_k)


def test_rule_of_the_backward_of_one_key_tile():
    assert one_kv(64, 1, 384, 128) and not one_kv(64, 1, 384, 129) and not one_kv(128, 512, 128, 128)
    assert not one_kv(64, 47, 385, 100) and one_kv(64, 48, 385, 100)      # four query tiles
    assert not one_kv(64, 59, 600, 100) and one_kv(64, 60, 600, 100)      # five

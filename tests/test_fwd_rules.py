"""The rule on sizes that picks the forward kernel of two query tiles per CTA, called in the built library (no GPU needed)."""
import ctypes as C

from nvfuserexamples_b200 import capi


def pair_pays(sms, heads, S_q, S_k):
    fn = capi.load()["_ZN4fmha13fwd_pair_paysEllll"]   # fmha::fwd_pair_pays(int64_t x 4)
    fn.argtypes, fn.restype = [C.c_int64] * 4, C.c_bool
    return fn(sms, heads, S_q, S_k)


def test_two_tile_rule():
    assert pair_pays(148, 64, 2048, 2048)       # 4 sequences of 16 heads: the shape the kernel was built for
    assert not pair_pays(148, 64, 2048, 256)    # two key steps
    assert not pair_pays(148, 64, 512, 2048)    # fewer than two query tiles per multiprocessor


def test_two_tile_rule_without_a_multiprocessor_count():
    """The number of multiprocessors is 0 where its query failed: the one-tile kernel, not a division by zero."""
    assert not pair_pays(0, 64, 2048, 2048)

"""The rules that choose slices for kernels, on the host."""
import pytest

from tiny_llm_b200 import ops


@pytest.mark.parametrize("head_dim", [64, 128])
@pytest.mark.parametrize("kv_heads", [1, 4, 8])
def test_slices_of_decoded_tokens_cover_every_tile_and_leave_none_empty(head_dim, kv_heads, monkeypatch):
    monkeypatch.setattr(ops, "sm_count", lambda *_: 148)
    per_tile = 4096 // head_dim
    for requests in (1, 2, 3, 8, 16, 19, 37, 64, 65, 149, 500):
        for keys in (1, 31, 32, 33, 64, 65, 300, 511, 512, 513, 1400, 2048, 3071, 3072, 3073, 6144, 6145, 8192, 100000):
            tiles, picked = -(-keys // per_tile), ops._decode_slices(requests, kv_heads, head_dim, keys)
            if picked is None:      # left to the kernel that cuts finer: SMs idle and slices are long
                assert requests * kv_heads * min(8, tiles) < 148 or requests * kv_heads * 7 < 148
                assert tiles > 12
                continue
            slices, few = picked
            per = -(-tiles // slices)
            assert 1 <= slices <= 8 and (slices - 1) * per < tiles <= slices * per
            assert per <= 8 if few else True


def test_slices_of_decoded_tokens_at_the_lines(monkeypatch):
    monkeypatch.setattr(ops, "sm_count", lambda *_: 148)
    pick = ops._decode_slices
    assert pick(1, 4, 64, 1) == (1, True) and pick(1, 4, 64, 300) == (2, True)          # one tile per warp at least
    assert pick(8, 4, 64, 1400) == (6, True) and pick(64, 4, 64, 300) == (1, True)      # at most eight tiles
    assert pick(64, 4, 64, 1400) == (1, False) and pick(16, 8, 128, 5600) == (2, False)
    assert pick(200, 8, 64, 2048) == (1, False)                                         # more items than CTAs fit
    assert pick(1, 8, 128, 3072) == (8, False) and pick(1, 8, 128, 3073) is None        # twelve tiles
    assert pick(1, 4, 64, 6144) == (8, False) and pick(1, 4, 64, 6145) is None
    assert pick(4, 8, 128, 5600) == (8, False)                                          # long slices, but no idle SM


def test_slices_of_32_bit_products(monkeypatch):
    """At most 296 CTAs, at least four blocks of 64 values each, whatever the part and the switches."""
    def pick(n, k):
        got = ops._f32_tc_slices(n, k)
        for split, sms in ((False, 148), (True, 40)):
            monkeypatch.setattr(ops, "split_k", split)
            monkeypatch.setattr(ops, "sm_count", lambda *_, sms=sms: sms)
            assert ops._f32_tc_slices(n, k) == got
        return got
    assert [pick(n, 2048) for n in (32, 2048, 2560, 4736, 4864, 9472, 9600, 18944, 18976, 32000)] == [8, 8, 8, 8, 4, 4, 2, 2, 1, 1]
    assert [pick(512, k) for k in (64, 256, 480, 512, 1024, 1984, 2048)] == [1, 1, 2, 2, 4, 4, 8]

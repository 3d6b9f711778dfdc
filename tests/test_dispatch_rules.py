"""The rules that choose between two forms of a kernel, at sizes where both were timed: a rule that sends a call to the slower form
fails here.  Host code only."""
import pytest

from infinicore_infer_b200.kernels import host


@pytest.mark.parametrize("heads,requests,window,keys", [
    # (rows, position of the first) of every request; microseconds on a B200 with tiles of 128 and of 64 keys
    (8, [(128, 4000)], 0, 128),                 # 72, 87
    (32, [(128, 4000)], 0, 128),                # 72, 88
    (64, [(128, 4000)], 0, 128),                # 73, 88
    (8, [(1000, 7000)], 0, 128),                # 125, 158
    (16, [(1024, 4000)], 0, 128),               # 87, 106
    (16, [(2048, 0)], 0, 128),                  # 45, 52
    (32, [(512, 0)], 0, 128),                   # 18, 20
    (32, [(1024, 0)], 0, 128),                  # 32, 34
    (32, [(1000, 0), (64, 3000)], 0, 128),      # 56, 72
    (32, [(1000, 0), (200, 0), (1, 3000)], 0, 64),      # the short request's row is no tile; 39, 34
    (16, [(2048, 4000)], 0, 64),                # 164, 138
    (16, [(2048, 0)], 1024, 64),                # 43, 37
    (16, [(1536, 0)], 512, 64),                 # 30, 26
    (32, [(768, 1000)], 0, 64),                 # 54, 50
    (32, [(1536, 0)], 0, 64),                   # 55, 48
    (32, [(100, 2000)] * 6, 0, 64),             # 81, 60
    (32, [(60, 0)] * 10, 0, 64),                # 28, 19
    (32, [(833, 0), (1667, 0), (2503, 0)], 0, 64)])     # 207, 152
def test_keys_a_tile_of_the_prefill_attention(heads, requests, window, keys):
    start = [0]
    for n, _ in requests:
        start.append(start[-1] + n)
    assert host.attention_tile_keys(heads, start, [p for _, p in requests], window) == keys

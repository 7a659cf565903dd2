"""The metadata block of a forward pass is filled sequence by sequence for few sequences and over all tokens for many: both ways give the same numbers."""
import random

import numpy as np
import pytest

from mistral_inference_b200.cache import BufferCache


@pytest.mark.parametrize("windows", [None, 4, [3, 9]])
def test_both_ways_of_filling_the_block_agree(windows):
    r = random.Random(0)
    for _ in range(120):
        B = r.choice([1, 2, 5, 16, 17, 30])
        cache = BufferCache(2, B, r.randint(2, 20), 1, 8, windows)
        cache.init_kvseqlens(B)
        if r.random() < 0.5:
            cache.update_seqlens([r.randint(1, 30) for _ in range(B)])
        lens = [r.randint(1, 12) if r.random() < 0.8 else 1 for _ in range(B)]
        host, layout = cache.build_metadata_host(lens)
        T, distinct = sum(lens), layout["windows"]
        for fill in (cache._fill_sequences, cache._fill_tokens):
            other = np.full_like(host, -7)
            fill(other, lens, T, distinct)
            assert (other == host).all()


@pytest.mark.parametrize("B,n,windows,by_sequence", [(1, 1, None, True), (5, 35, None, True), (8, 1, None, False), (16, 1, None, False), (16, 400, None, True), (3, 1, 64, True),
                                                     (4, 1, 64, False), (2, 1, [16, 64, 4096], True), (16, 35, [64, 4096], False)])
def test_the_cheaper_way_is_taken(B, n, windows, by_sequence):
    cache = BufferCache(len(windows) if isinstance(windows, list) else 1, B, 4200, 1, 8, windows)
    cache.init_kvseqlens(B)
    cache.update_seqlens([100] * B)
    taken = []
    for name in ("_fill_sequences", "_fill_tokens"):
        setattr(cache, name, lambda *a, name=name: taken.append(name))
    cache.build_metadata_host([n] * B)
    assert taken == ["_fill_sequences" if by_sequence else "_fill_tokens"]

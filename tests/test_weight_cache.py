"""The weight cache's native host logic (no GPU)."""
import torch

import nanochat_cpp_b200 as nc


def test_a_new_weight_is_never_taken_for_a_dead_one():
    """A dead tensor's addresses are reused at once; a new weight there has the old one's version too."""
    cache = nc.Fp8WeightCache(True)
    for i in range(50):
        w = torch.full((128, 128), float(i))
        assert cache.get(1, [w], lambda: [w.clone()])[0][0, 0] == i
        del w


def test_a_weight_under_another_name_and_another_kind():
    cache = nc.Fp8WeightCache(True)
    w, v = torch.zeros(128, 128), torch.ones(128, 128)
    first = cache.get(1, [w, v], lambda: [1])
    assert cache.get(1, [w, v], lambda: [2]) is first
    assert cache.get(2, [w, v], lambda: [3]) == [3]
    assert cache.get(2, [v, w], lambda: [4]) == [4]
    assert cache.get(2, [w.view(128, 128), w], lambda: [5]) == [5]
    assert cache.get(2, [w], lambda: [6]) == [6]

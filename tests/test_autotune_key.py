"""The autotuner's cache key: a shape tuned for millions of rays is not applied to
a call of a thousand."""
import types

import numpy as np

import cubiquity_gb300 as cbq
from cubiquity_gb300 import autotune


def test_key_has_the_ray_count_class():
    dag = types.SimpleNamespace(bytes=1 << 20, layout=cbq.LAYOUT_REFERENCE)
    d = np.tile(np.array([[0.5, 0.5, 0.7, 0.0]], np.float32), (1 << 20, 1))
    keys = {n: autotune.cache_key(dag, d[:n]) for n in (1, 1000, 1024, 1100, 100_000, 1_000_000, 1 << 20)}
    assert keys[1000] == keys[1024] == keys[1100] and keys[1_000_000] == keys[1 << 20]
    assert len(set(keys.values())) == 4
    assert autotune.cache_key(dag, d[:0])

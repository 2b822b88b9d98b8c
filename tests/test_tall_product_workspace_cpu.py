"""A workspace sized for a tall product serves every smaller one too: callers size
it once for the largest of their calls."""
import random

from capytaine_b200 import _lib


def test_workspace_grows_with_every_size():
    size = _lib.load().bem_zgemm_ts_workspace_bytes
    assert size(129, 10000, 1, 1) >= size(128, 10000, 1, 1)
    rng = random.Random(4)
    for _ in range(4000):
        big = [int(10 ** rng.uniform(0, top)) for top in (4.5, 4.5, 1.2, 1.8)]
        small = [rng.choice([b, max(1, b - 1), rng.randint(1, b)]) for b in big]
        assert size(*big) >= size(*small) > 0, (big, small)
        assert size(*big) >= 16 * big[0] * big[2] * big[3]

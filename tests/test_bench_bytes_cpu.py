"""CPU test of the bench's byte model of the extension: what a pass reads and
writes once, whatever the tiles of hits that it does not scan."""
import bench


def test_extension_bytes():
    st = {"seeds_with_hits": 10, "num_hits": 1000, "num_hsps": 7, "tiles": 5000, "survivors": 300}
    want = 24 * 10 + 4 * 1000 + 50 + 2 * 30 + 16 * 7
    assert bench.extension_bytes(st, 100, 60) == want
    assert bench.extension_bytes({**st, "tiles": 10**9, "survivors": 10**6}, 100, 60) == want

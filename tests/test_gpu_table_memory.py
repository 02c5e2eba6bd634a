"""GPU test of a seed-table build that finds no device memory: it reports that,
and the table there was goes on serving calls."""
import numpy as np
import pytest

from segalign_b200 import SegAlignError, SeedFilter, build_sub_mat, host_seeds
from tests.helpers import compare_segments, random_text

pytestmark = pytest.mark.gpu


def test_failed_build_keeps_the_table(built):
    import torch
    rng = np.random.default_rng(61)
    T = random_text(rng, 40_000_000)
    Q = random_text(rng, 3000) + T[5000:9000] + random_text(rng, 3000)
    sf = SeedFilter()
    sf.initialize_interface(1)
    sf.generate_shape_pos("12of19")
    sf.initialize_processor(False, 20_000, 19, build_sub_mat(910), 910, 3000, False)
    sf.send_ref_write_request(T)
    sf.send_query_write_request(Q, 0)
    sf.generate_seed_pos_table(None, 20, 19, 12)
    seeds = host_seeds(Q, 0, len(Q) - 19)
    want, table = sf.seed_and_filter(seeds, False, 0), sf.get_seed_pos_table()
    # step 1 takes 640 MB (keys, positions, both twice)
    filler = torch.empty(torch.cuda.mem_get_info()[0] - (300 << 20), dtype=torch.uint8, device="cuda")
    try:
        with pytest.raises(SegAlignError) as ei:
            sf.generate_seed_pos_table(None, 1, 19, 12)
        assert ei.value.code == -4  # SA_ERR_NOMEM
        assert all(np.array_equal(a, b) for a, b in zip(sf.get_seed_pos_table(), table))
        compare_segments(sf.seed_and_filter(seeds, False, 0), want, "after the failed build")
    finally:
        del filler
        torch.cuda.empty_cache()
    sf.generate_seed_pos_table(None, 1, 19, 12)
    assert len(sf.get_seed_pos_table()[1]) > 10 * len(table[1])
    sf.clear_ref()

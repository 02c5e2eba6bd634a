"""GPU test of what the autotuner searches and reuses: only knobs that act on the
kernels the scores lead to, and no settings timed on other kernels."""
import json
import re

import pytest

from segalign_b200 import SeedFilter, build_sub_mat
from tests.helpers import small_workload

pytestmark = pytest.mark.gpu

QUICK = {"step_bases": (16, 32), "lane_cap": (2048, 4096), "range_ctas": (296,), "substeps": (2, 3)}
LANE_ONLY = {"ext_ctas_per_sm": (2, 3), "tile_hits": (128, 160, 224), "switch_now": (0, 1)}


@pytest.mark.parametrize("xdrop,knobs", [(910, QUICK), (699, {**QUICK, **LANE_ONLY})])  # below 7 matches: no sweep
def test_knobs_and_cache(built, tmp_path, xdrop, knobs):
    w = small_workload(0.25)
    sf = SeedFilter()
    sf.initialize_interface(1)
    sf.generate_shape_pos("12of19")
    sf.initialize_processor(False, 250_000, 19, build_sub_mat(xdrop), xdrop, 3000, False)
    sf.send_ref_write_request(w.target)
    sf.generate_seed_pos_table(None, 1, 19, 12)
    sf.send_query_write_request(w.query, 0)
    saved = sf.get_tuning()
    units = [(0, r, a, a + 50_000) for r in (0, 1) for a in (0, 50_000, 100_000)]
    cache = tmp_path / "tune.jsonl"
    try:
        res = sf.autotune(units, cache_path=str(cache), quick=True, repeats=1)
        assert res["candidates"] == sum(v != saved[k] for k, vs in knobs.items() for v in vs)
        for k in LANE_ONLY:
            if k not in knobs:
                assert res[k] == saved[k]
        # a line of a build that did not name its kernels
        line = json.loads(cache.read_text())
        line["key"] = re.sub(r"\|kernels=\d+", "", line["key"])
        cache.write_text(json.dumps(line) + "\n")
        sf.set_tuning(**saved)
        assert sf.autotune(units, cache_path=str(cache), quick=True, repeats=1)["from_cache"] == 0
    finally:
        sf.set_tuning(**saved)
